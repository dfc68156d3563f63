// Airwave top boundary in complex64 (airbc_init_free.c:130-209) in three kernels, for uniform
// grids of 64, 256 or 1024 points a side that have more rows than the model.
//
// Hz(z=0) is interpolated from the stretched grid (n1 x n2) to the uniform one (N1 x N2),
// Fourier transformed, multiplied by two filters, transformed back and interpolated to the
// ghosts' nodes. The interpolations are products of one in x and one in y, and each commutes
// with the transform along the other axis. So the transforms along x only run over the
// model's n2 rows, not the uniform grid's N2, and nothing of the uniform grid's size is ever
// stored:
//   k_air_rows     Hz of a row, interpolated along x, transformed along x
//   k_air_columns  interpolated along y, transformed along y, times a filter, back along y,
//                  interpolated to the ghosts' rows (both filters)
//   k_air_ghosts   back along x, interpolated to the ghosts' nodes
// 200 x 140 model, 1024^2 grid: 7 MB of memory traffic a system besides the filters (shared,
// in L2), against 130 MB for two-dimensional transforms of the interpolated grid.
//
// A transform of N = A^2 points runs in A lanes: lane b takes the points A a + b, does an
// A-point transform over a in registers, turns the A x A values in shared memory and does a
// second one (the four-step method; D. H. Bailey, J. Supercomputing 4, 1990).
//
// 16 systems, 200 x 140 model, 1024^2 grid: rows 13 us, columns 118 us, ghosts 18 us, against
// some 500 us for the interpolated grid through two-dimensional transforms (the operator, alone:
// 1335 -> 978 us; 3 small systems 173 -> 75 us). The columns are bound by issue: three
// transforms of 1024 points are 6000 instructions a warp, at 12 warps an SM (168 registers: the
// spectrum is kept over the two filters).
#include <cmath>
#include "csem_cuda.cuh"
#include "engine.h"

namespace csem {

namespace {

typedef float2 C;

__device__ __forceinline__ C mul(C a, C b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ C lerp(C a, C b, float w) { return make_float2((1.f - w) * a.x + w * b.x, (1.f - w) * a.y + w * b.y); }

// cos(2 pi k / 32)
__host__ __device__ constexpr float cos32(int k)
{
  k &= 31;
  if (k > 16) k = 32 - k;
  const float s = k > 8 ? -1.f : 1.f;
  if (k > 8) k = 16 - k;
  constexpr float c[9] = {1.f,
                          0.98078528040323044913f,
                          0.92387953251128675613f,
                          0.83146961230254523708f,
                          0.70710678118654752440f,
                          0.55557023301960222474f,
                          0.38268343236508977173f,
                          0.19509032201612826785f,
                          0.f};
  return s * c[k];
}
__host__ __device__ constexpr int reversed(int k, int A)
{
  int r = 0;
  for (int b = 1; b < A; b <<= 1) r = r * 2 + ((k & b) ? 1 : 0);
  return r;
}

// A-point transform in registers, frequency k at place reversed(k, A)
template <int A, bool INV> __device__ __forceinline__ void dft(C (&x)[A])
{
#pragma unroll
  for (int len = A; len >= 2; len /= 2) {
#pragma unroll
    for (int p = 0; p < A / 2; p++) {
      const int k = p % (len / 2), a = p / (len / 2) * len + k, b = a + len / 2;
      const C u = x[a], v = x[b];
      x[a] = make_float2(u.x + v.x, u.y + v.y);
      const C d = make_float2(u.x - v.x, u.y - v.y);
      const int t = k * (32 / len);  // times exp(-+2 pi i t / 32)
      if (t == 0) x[b] = d;
      else if (t == 8) x[b] = INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
      else x[b] = mul(d, make_float2(cos32(t), INV ? cos32(t - 8) : -cos32(t - 8)));
    }
  }
}

// x[a] = point A a + lane on entry; frequency (or point) lane + A d at x[reversed(d, A)] after.
// tw[c A + b] = exp(-2 pi i b c / A^2); buf: A (A + 1) of this group of A lanes
template <int A, bool INV> __device__ __forceinline__ void fft(C (&x)[A], const C* __restrict__ tw, C* buf, int b)
{
  dft<A, INV>(x);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < A; c++) {
    C t = __ldg(tw + c * A + b);
    if (INV) t.y = -t.y;
    buf[c * (A + 1) + b] = c == 0 ? x[0] : mul(x[reversed(c, A)], t);
  }
  __syncwarp();
#pragma unroll
  for (int a = 0; a < A; a++) x[a] = buf[b * (A + 1) + a];
  dft<A, INV>(x);
}

template <int A> constexpr int GROUPS = 128 / A;  // groups of A lanes (rows, columns) of a CTA

}  // namespace

// grid (rows, slots) in groups of A lanes; T [slot][n2][N1]. Shared: per group n1 Hz values
// and A (A + 1)
template <int A>
__global__ void __launch_bounds__(128) k_air_rows(GridP<F32> g, AirP<F32> a, const SysScal<F32>* scal, const C* X,
                                                  const int* sys_list, const C* tw, C* T)
{
  extern __shared__ C smem[];
  constexpr int G = GROUPS<A>;
  const int grp = threadIdx.x / A, b = threadIdx.x % A;
  const int j = min(blockIdx.x * G + grp, a.n2 - 1), slot = blockIdx.y;
  const int sys = sys_list ? sys_list[slot] : slot;
  const int n1 = a.n1;
  C* hz = smem + grp * (n1 + A * (A + 1));
  C* buf = hz + n1;
  const C* Ex = X + (size_t)sys * g.lE + (long)j * n1;
  const C* Ey = X + (size_t)sys * g.lE + g.lEx + (long)j * (n1 + 1);
  const C iwmu = scal[sys].iwmu;
  const float r2s = g.r2s[j];
  for (int i = b; i < n1; i += A) {  // Hz = (dEy/dx - dEx/dy) / (i w mu0)
    const float r1s = g.r1s[i];
    const C e0 = Ey[i], e1 = Ey[i + 1], f0 = Ex[i], f1 = Ex[i + n1];
    hz[i] = mul(make_float2((e1.x - e0.x) * r1s - (f1.x - f0.x) * r2s, (e1.y - e0.y) * r1s - (f1.y - f0.y) * r2s), iwmu);
  }
  __syncwarp();
  C x[A];
#pragma unroll
  for (int q = 0; q < A; q++) {
    const int u = q * A + b, jx = a.jx[u];
    x[q] = jx >= 0 ? lerp(hz[jx], hz[jx + 1], a.wx[u]) : make_float2(0.f, 0.f);
  }
  fft<A, false>(x, tw, buf, b);
  C* out = T + ((size_t)slot * a.n2 + j) * a.N1;
#pragma unroll
  for (int d = 0; d < A; d++) out[b + A * d] = x[reversed(d, A)];
}

// One frequency of x per group of A lanes. grid (N1 / groups, slots). T1 [slot][n2][N1], T2
// [slot][n2 + 1][N1]; the filters transposed, [N1][N2]. Shared: n2 + 1 rows of the columns, and
// per column A (A + 1) + 1
template <int A>
__global__ void __launch_bounds__(128, 3) k_air_columns(AirP<F32> a, const C* tw, const C* T, C* T1, C* T2)
{
  extern __shared__ C smem[];
  constexpr int COLS = GROUPS<A>;
  const int col = threadIdx.x / A, b = threadIdx.x % A;
  const int c0 = blockIdx.x * COLS, slot = blockIdx.y;
  const int n2 = a.n2, N1 = a.N1, N2 = a.N2;
  C* tile = smem;                                        // [rows][COLS]
  C* buf = smem + (n2 + 1) * COLS + col * (A * (A + 1) + 1);  // (odd: the columns on different banks)
  const C* in = T + (size_t)slot * n2 * N1 + c0;
  for (int q = threadIdx.x; q < n2 * COLS; q += 128) tile[q] = in[(size_t)(q / COLS) * N1 + q % COLS];
  __syncthreads();
  C x[A];
#pragma unroll
  for (int q = 0; q < A; q++) {
    const int u = q * A + b, jy = a.jy[u];
    x[q] = jy >= 0 ? lerp(tile[jy * COLS + col], tile[(jy + 1) * COLS + col], a.wy[u]) : make_float2(0.f, 0.f);
  }
  fft<A, false>(x, tw, buf, b);
#pragma unroll 1
  for (int f = 0; f < 2; f++) {
    const C* H = (f ? a.sH2 : a.sH1) + (size_t)(c0 + col) * N2;
    C y[A];
#pragma unroll
    for (int q = 0; q < A; q++) y[q] = mul(x[reversed(q, A)], __ldg(H + b + A * q));  // frequency A q + b
    fft<A, true>(y, tw, buf, b);
    __syncwarp();
#pragma unroll
    for (int d = 0; d < A; d++) buf[b + A * d] = y[reversed(d, A)];
    __syncthreads();  // (the tile's earlier use is over, too)
    const int rows = n2 + f;
    const int* j2 = f ? a.hy_j2 : a.hx_j2;
    const float* w2 = f ? a.hy_w2 : a.hx_w2;
    for (int r = b; r < rows; r += A) {
      const int q = j2[r];
      const C lo = buf[q], hi = q + 1 < N2 ? buf[q + 1] : make_float2(0.f, 0.f);  // past the last node: zero
      tile[r * COLS + col] = lerp(lo, hi, w2[r]);
    }
    __syncthreads();
    C* out = (f ? T2 + (size_t)slot * (n2 + 1) * N1 : T1 + (size_t)slot * n2 * N1) + c0;
    for (int q = threadIdx.x; q < rows * COLS; q += 128) out[(size_t)(q / COLS) * N1 + q % COLS] = tile[q];
  }
}

// rows 0..n2-1: Hx's ghosts from T1, n2..2 n2: Hy's from T2. grid (rows, slots) in groups of A
// lanes. Shared: per group A (A + 1)
template <int A>
__global__ void __launch_bounds__(128) k_air_ghosts(AirP<F32> a, const C* tw, const C* T1, const C* T2, C* ghx, C* ghy)
{
  extern __shared__ C smem[];
  constexpr int G = GROUPS<A>;
  const int grp = threadIdx.x / A, b = threadIdx.x % A;
  const int n1 = a.n1, n2 = a.n2, N1 = a.N1, slot = blockIdx.y;
  const int row = min(blockIdx.x * G + grp, 2 * n2);
  C* buf = smem + grp * (A * (A + 1));
  const bool hy = row >= n2;
  const int j = hy ? row - n2 : row;
  const C* in = hy ? T2 + ((size_t)slot * (n2 + 1) + j) * N1 : T1 + ((size_t)slot * n2 + j) * N1;
  C x[A];
#pragma unroll
  for (int q = 0; q < A; q++) x[q] = in[A * q + b];
  fft<A, true>(x, tw, buf, b);
  __syncwarp();
  const float s = 1.f / ((float)N1 * (float)a.N2);
#pragma unroll
  for (int d = 0; d < A; d++) {
    const C v = x[reversed(d, A)];
    buf[b + A * d] = make_float2(s * v.x, s * v.y);
  }
  __syncwarp();
  const int n = hy ? n1 : n1 + 1;
  const int* j1 = hy ? a.hy_j1 : a.hx_j1;
  const float* w1 = hy ? a.hy_w1 : a.hx_w1;
  C* out = hy ? ghy + ((size_t)slot * (n2 + 1) + j) * n1 : ghx + ((size_t)slot * n2 + j) * (n1 + 1);
  for (int i = b; i < n; i += A) {
    const int q = j1[i];
    out[i] = lerp(buf[q], q + 1 < N1 ? buf[q + 1] : make_float2(0.f, 0.f), w1[i]);
  }
}

static int side(int N) { return N == 64 ? 8 : (N == 256 ? 16 : (N == 1024 ? 32 : 0)); }
static size_t rows_smem(int A, int n1) { return (size_t)(128 / A) * (n1 + A * (A + 1)) * 8; }
static size_t columns_smem(int A, int n2) { return (size_t)(128 / A) * (n2 + 1 + A * (A + 1) + 1) * 8; }

// Square grids: of others the two-dimensional transforms reproduce the reference's, which takes
// n1fft for the slow axis (airbc_init_free.c:48-49 plans n1fft x n2fft; the data is n2fft rows of n1fft).
// Fewer rows than the uniform grid's, so that the buffers are the smaller ones; two CTAs per SM.
bool airwave32_fits(int n1, int n2, int N1, int N2)
{
  const int A = side(N1);
  return A && N1 == N2 && n2 < N2 && rows_smem(A, n1) <= 113 * 1024 && columns_smem(A, n2) <= 113 * 1024;
}

std::vector<float2> air_twiddles(int N)
{
  std::vector<float2> t((size_t)N);
  const int A = side(N);
  for (int c = 0; c < A; c++)
    for (int b = 0; b < A; b++) {
      const double th = -2.0 * M_PI * b * c / N;
      t[(size_t)c * A + b] = make_float2((float)cos(th), (float)sin(th));
    }
  return t;
}

template <int A>
static void launch_air(const GridP<F32>& g, const AirP<F32>& a, const SysScal<F32>* scal, const C* X, const int* sys_list,
                       const C* tw, C* T, C* T12, C* ghx, C* ghy, int nslot, cudaStream_t st)
{
  constexpr int G = GROUPS<A>;
  C *T1 = T12, *T2 = T12 + (size_t)nslot * a.n2 * a.N1;
  const size_t sr = rows_smem(A, a.n1), sc = columns_smem(A, a.n2);
  allow_smem<k_air_rows<A>>(sr);
  allow_smem<k_air_columns<A>>(sc);
  count_launch(), k_air_rows<A><<<dim3((a.n2 + G - 1) / G, nslot), 128, sr, st>>>(g, a, scal, X, sys_list, tw, T);
  count_launch(), k_air_columns<A><<<dim3(a.N1 / G, nslot), 128, sc, st>>>(a, tw, T, T1, T2);
  count_launch(), k_air_ghosts<A><<<dim3((2 * a.n2 + G) / G, nslot), 128, (size_t)G * A * (A + 1) * 8, st>>>(a, tw, T1, T2, ghx, ghy);
}

void launch_airwave32(const GridP<F32>& g, const AirP<F32>& a, const SysScal<F32>* scal, const C* X, const int* sys_list,
                      const C* tw, C* T, C* T12, C* ghx, C* ghy, int nslot, cudaStream_t st)
{
  switch (side(a.N1)) {
    case 8: return launch_air<8>(g, a, scal, X, sys_list, tw, T, T12, ghx, ghy, nslot, st);
    case 16: return launch_air<16>(g, a, scal, X, sys_list, tw, T, T12, ghx, ghy, nslot, st);
    default: return launch_air<32>(g, a, scal, X, sys_list, tw, T, T12, ghx, ghy, nslot, st);
  }
}

}  // namespace csem
