"""Error of the quick complex128 operator (csrc/k_fdfd.cu, the batched solver's outer residuals)
against 64-bit-mantissa arithmetic or better, beside that of the operator with the reference's bits.

1 / (i omega mu0) divided by a spacing carries one rounding, the same in all of a column's or
plane's points, where the reference divides by the spacing and multiplies by it, two roundings
that differ from point to point; the rest is as many roundings in both, or fewer (multiply-adds).
So over models whose spacings and frequencies differ the quick operator's error is the other's, up
to the models' scatter, some tenth each: the geometric mean over 24 of them within 5%."""
import os
import subprocess

import pytest

from demo_matrixfree_csem_gb300 import build as b

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "csem_gpu.h"
#include "csem_host.h"
#include "engine_model.h"
using namespace csem;
typedef long double L;
struct Z { L x, y; };
static Z operator-(Z a, Z b) { return {a.x - b.x, a.y - b.y}; }
static Z operator*(L s, Z a) { return {s * a.x, s * a.y}; }
static Z operator/(Z a, L s) { return {a.x / s, a.y / s}; }
int main()
{
  double sum = 0;
  const int models = 24;
  for (int c = 0; c < models; c++) {
    std::mt19937 g(c + 1);
    std::normal_distribution<double> N;
    const int n[3] = {12 + 2 * (c % 5), 11 + 3 * (c % 4), 10 + 2 * (c % 3)}, fvm = c & 1;
    std::vector<float> x[3], rho((size_t)n[0] * n[1] * n[2]);
    for (int a = 0; a < 3; a++) {
      const float h = 40.f + g() % 3000 * 0.1f;
      for (int i = 0; i <= n[a]; i++) x[a].push_back(i * h);
    }
    const double w = 2 * M_PI * (0.1 + g() % 2000 * 0.001) * 4e-7 * M_PI;
    for (auto& r : rho) r = 0.5f + (g() % 1000) * 0.01f;
    csem_grid_t G = {};
    csem_grid_set(&G, n[0], n[1], n[2], x[0].data(), x[1].data(), x[2].data(), rho.data(), rho.data(), rho.data());
    csem_grid_extend(&G, 4, 4e3f, 1e6f, 1);
    Model m((const csem_grid*)&G, 0, fvm);
    Ops<F64> o(&m, 1, 0);
    std::vector<double2> in(m.lE), y[2];
    for (auto& v : in) v = make_double2(N(g), N(g));
    DevBuf X, Y, S;
    X.alloc(16 * m.lE), Y.alloc(16 * m.lE), S.alloc(64);
    const SysScal<F64> s = sys_scal64(0, w);
    cudaMemcpy(S.p, &s, sizeof(s), cudaMemcpyHostToDevice);
    cudaMemcpy(X.p, in.data(), 16 * m.lE, cudaMemcpyHostToDevice);
    for (int q = 0; q < 2; q++) {
      y[q].resize(m.lE);
      o.quick_stencil = q != 0;
      o.apply_A(X.as<double2>(), Y.as<double2>(), 1, nullptr, S.as<SysScal<F64>>());
      if (cudaMemcpy(y[q].data(), Y.p, 16 * m.lE, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    }
    const int n1 = m.n1, n2 = m.n2, n3 = m.n3;
    auto E = [&](int a, int k, int j, int i) {
      const long at = a == 0 ? (long)n1 * (j + (long)(n2 + 1) * k) + i
                             : (a == 1 ? m.lEx + (long)(n1 + 1) * (j + (long)n2 * k) + i : m.lEx + m.lEy + (long)(n1 + 1) * (j + (long)(n2 + 1) * k) + i);
      return at;
    };
    auto e = [&](int a, int k, int j, int i) { const double2 v = in[E(a, k, j, i)]; return Z{v.x, v.y}; };
    auto over = [&](Z t) { return Z{t.y / (L)w, -t.x / (L)w}; };  // by i w
    auto hx = [&](int k, int j, int i) { return over((e(2, k, j + 1, i) - e(2, k, j, i)) / (L)G.d2s[j] - (e(1, k + 1, j, i) - e(1, k, j, i)) / (L)G.d3s[k]); };
    auto hy = [&](int k, int j, int i) { return over((e(0, k + 1, j, i) - e(0, k, j, i)) / (L)G.d3s[k] - (e(2, k, j, i + 1) - e(2, k, j, i)) / (L)G.d1s[i]); };
    auto hz = [&](int k, int j, int i) { return over((e(1, k, j, i + 1) - e(1, k, j, i)) / (L)G.d1s[i] - (e(0, k, j + 1, i) - e(0, k, j, i)) / (L)G.d2s[j]); };
    L err[2] = {0, 0};
    auto point = [&](int a, int k, int j, int i, Z v, double sigma, double vol) {
      v = v - (L)sigma * e(a, k, j, i);
      if (fvm) v = (L)vol * (L)w * Z{-v.y, v.x};
      for (int q = 0; q < 2; q++) {
        const double2 r = y[q][E(a, k, j, i)];
        err[q] += (r.x - v.x) * (r.x - v.x) + (r.y - v.y) * (r.y - v.y);
      }
    };
    for (int k = 1; k < n3; k++)
      for (int j = 1; j < n2; j++)
        for (int i = 1; i < n1; i++) {
          const L d1 = G.d1[i], d2 = G.d2[j], d3 = G.d3[k];
          point(0, k, j, i, (hz(k, j, i) - hz(k, j - 1, i)) / d2 - (hy(k, j, i) - hy(k - 1, j, i)) / d3, G.sigma11[E(0, k, j, i)], G.d1s[i] * d2 * d3);
          point(1, k, j, i, (hx(k, j, i) - hx(k - 1, j, i)) / d3 - (hz(k, j, i) - hz(k, j, i - 1)) / d1, G.sigma22[E(1, k, j, i) - m.lEx], d1 * G.d2s[j] * d3);
          point(2, k, j, i, (hy(k, j, i) - hy(k, j, i - 1)) / d1 - (hx(k, j, i) - hx(k, j - 1, i)) / d2, G.sigma33[E(2, k, j, i) - m.lEx - m.lEy], d1 * d2 * G.d3s[k]);
        }
    sum += std::log(std::sqrt((double)(err[1] / err[0])));
    csem_grid_free(&G);
  }
  printf("%.4f\n", std::exp(sum / models));
}
"""


def test_error_of_the_quick_operator(gpu, tmp_path):
    src, exe = tmp_path / "quick.cu", tmp_path / "quick"
    src.write_text(PROGRAM)
    subprocess.run([b.NVCC, *b.ARCH, "-O1", "-std=c++17", "--cudart", "shared", "-I", b.INCLUDE, "-I", b.CSRC, str(src), "-o", str(exe),
                    f"-L{b.OUT}", "-lcsem_gpu", "-Xlinker", f"-rpath={b.OUT}", "-Xlinker", f"-rpath={os.path.join(b.CUDA_HOME, 'lib64')}"],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert abs(float(r.stdout) - 1) <= 0.05, r.stdout
