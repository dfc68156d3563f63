// Airwave top boundary (airbc_init_free.c:130-209) in three kernels, for uniform grids of 64, 256
// or 1024 points a side that have more rows than the model: in complex64, and in complex128 where
// the bits of the reference's transforms do not count (the batched solver's outer residuals).
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
// 200 x 140 model, 1024^2 grid, complex64: 7 MB of memory traffic a system besides the filters
// (shared, in L2), against 130 MB for two-dimensional transforms of the interpolated grid.
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
// complex128, 24 systems: 12.2 -> 6.0 ms (columns 5.2, ghosts 0.5, rows 0.3), bound by 3500 FP64
// operations a lane and column at 2 per SM and cycle.
#include <cmath>
#include "csem_cuda.cuh"
#include "engine.h"

namespace csem {

namespace {

template <class P> using Cx = typename P::C;
template <class P> using Re = typename P::R;
template <class P> __device__ __forceinline__ Cx<P> cx(Re<P> x, Re<P> y)
{
  Cx<P> c;
  c.x = x;
  c.y = y;
  return c;
}
template <class P> __device__ __forceinline__ Cx<P> mul(Cx<P> a, Cx<P> b)
{
  return cx<P>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class P> __device__ __forceinline__ Cx<P> lerp(Cx<P> a, Cx<P> b, Re<P> w)
{
  return cx<P>((1 - w) * a.x + w * b.x, (1 - w) * a.y + w * b.y);
}

// cos(2 pi k / 32)
template <class R> __host__ __device__ constexpr R cos32(int k)
{
  k &= 31;
  if (k > 16) k = 32 - k;
  const R s = k > 8 ? R(-1) : R(1);
  if (k > 8) k = 16 - k;
  constexpr R c[9] = {R(1),
                          R(0.98078528040323044913),
                          R(0.92387953251128675613),
                          R(0.83146961230254523708),
                          R(0.70710678118654752440),
                          R(0.55557023301960222474),
                          R(0.38268343236508977173),
                          R(0.19509032201612826785),
                          R(0)};
  return s * c[k];
}
__host__ __device__ constexpr int reversed(int k, int A)
{
  int r = 0;
  for (int b = 1; b < A; b <<= 1) r = r * 2 + ((k & b) ? 1 : 0);
  return r;
}

// A-point transform in registers, frequency k at place reversed(k, A)
template <class P, int A, bool INV> __device__ __forceinline__ void dft(Cx<P> (&x)[A])
{
#pragma unroll
  for (int len = A; len >= 2; len /= 2) {
#pragma unroll
    for (int p = 0; p < A / 2; p++) {
      const int k = p % (len / 2), a = p / (len / 2) * len + k, b = a + len / 2;
      const Cx<P> u = x[a], v = x[b];
      x[a] = cx<P>(u.x + v.x, u.y + v.y);
      const Cx<P> d = cx<P>(u.x - v.x, u.y - v.y);
      const int t = k * (32 / len);  // times exp(-+2 pi i t / 32)
      if (t == 0) x[b] = d;
      else if (t == 8) x[b] = INV ? cx<P>(-d.y, d.x) : cx<P>(d.y, -d.x);
      else x[b] = mul<P>(d, cx<P>(cos32<Re<P>>(t), INV ? cos32<Re<P>>(t - 8) : -cos32<Re<P>>(t - 8)));
    }
  }
}

// x[a] = point A a + lane on entry; frequency (or point) lane + A d at x[reversed(d, A)] after.
// tw[c A + b] = exp(-2 pi i b c / A^2); buf: A (A + 1) of this group of A lanes
template <class P, int A, bool INV>
__device__ __forceinline__ void fft(Cx<P> (&x)[A], const Cx<P>* __restrict__ tw, Cx<P>* buf, int b)
{
  dft<P, A, INV>(x);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < A; c++) {
    Cx<P> t = __ldg(tw + c * A + b);
    if (INV) t.y = -t.y;
    buf[c * (A + 1) + b] = c == 0 ? x[0] : mul<P>(x[reversed(c, A)], t);
  }
  __syncwarp();
#pragma unroll
  for (int a = 0; a < A; a++) x[a] = buf[b * (A + 1) + a];
  dft<P, A, INV>(x);
}

template <int A> constexpr int GROUPS = 128 / A;  // groups of A lanes (rows) of a CTA
// k_air_columns: threads of a CTA, and whether the spectrum is kept in shared memory over the two
// filters (complex128, whose two sets of values do not fit the registers)
template <class P> constexpr int COL_THREADS = sizeof(Re<P>) == 4 ? 128 : 64;
template <class P> constexpr bool SPECTRUM = sizeof(Re<P>) == 8;

}  // namespace

// grid (rows, slots) in groups of A lanes; T [slot][n2][N1]. Shared: per group n1 Hz values
// and A (A + 1)
template <class P, int A>
__global__ void __launch_bounds__(128) k_air_rows(GridP<P> g, AirP<P> a, const SysScal<P>* scal, const Cx<P>* X,
                                                  const int* sys_list, const Cx<P>* tw, Cx<P>* T)
{
  extern __shared__ char raw[];
  Cx<P>* const smem = (Cx<P>*)raw;
  constexpr int G = GROUPS<A>;
  const int grp = threadIdx.x / A, b = threadIdx.x % A;
  const int j = min(blockIdx.x * G + grp, a.n2 - 1), slot = blockIdx.y;
  const int sys = sys_list ? sys_list[slot] : slot;
  const int n1 = a.n1;
  Cx<P>* hz = smem + grp * (n1 + A * (A + 1));
  Cx<P>* buf = hz + n1;
  const Cx<P>* Ex = X + (size_t)sys * g.lE + (long)j * n1;
  const Cx<P>* Ey = X + (size_t)sys * g.lE + g.lEx + (long)j * (n1 + 1);
  const Cx<P> iwmu = scal[sys].iwmu;
  const Re<P> r2s = g.r2s[j];
  for (int i = b; i < n1; i += A) {  // Hz = (dEy/dx - dEx/dy) / (i w mu0)
    const Re<P> r1s = g.r1s[i];
    const Cx<P> e0 = Ey[i], e1 = Ey[i + 1], f0 = Ex[i], f1 = Ex[i + n1];
    hz[i] = mul<P>(cx<P>((e1.x - e0.x) * r1s - (f1.x - f0.x) * r2s, (e1.y - e0.y) * r1s - (f1.y - f0.y) * r2s), iwmu);
  }
  __syncwarp();
  Cx<P> x[A];
#pragma unroll
  for (int q = 0; q < A; q++) {
    const int u = q * A + b, jx = a.jx[u];
    x[q] = jx >= 0 ? lerp<P>(hz[jx], hz[jx + 1], a.wx[u]) : cx<P>(0, 0);
  }
  fft<P, A, false>(x, tw, buf, b);
  Cx<P>* out = T + ((size_t)slot * a.n2 + j) * a.N1;
#pragma unroll
  for (int d = 0; d < A; d++) out[b + A * d] = x[reversed(d, A)];
}

// One frequency of x per group of A lanes. grid (N1 / groups, slots). T1 [slot][n2][N1], T2
// [slot][n2 + 1][N1]; the filters [N1][N2] in complex64, [N2][N1] in
// complex128 (two columns are a sector). Shared: n2 + 1 rows of the
// columns, per column A (A + 1) + 1, and the spectra
template <class P, int A>
__global__ void __launch_bounds__(COL_THREADS<P>, 3)
    k_air_columns(AirP<P> a, const Cx<P>* tw, const Cx<P>* T, Cx<P>* T1, Cx<P>* T2)
{
  extern __shared__ char raw[];
  Cx<P>* const smem = (Cx<P>*)raw;
  constexpr int TH = COL_THREADS<P>, COLS = TH / A;
  const int col = threadIdx.x / A, b = threadIdx.x % A;
  const int c0 = blockIdx.x * COLS, slot = blockIdx.y;
  const int n2 = a.n2, N1 = a.N1, N2 = a.N2;
  Cx<P>* tile = smem;                                             // [rows][COLS]
  Cx<P>* buf = smem + (n2 + 1) * COLS + col * (A * (A + 1) + 1);  // (odd: the columns on different banks)
  Cx<P>* spec = smem + (n2 + 1) * COLS + COLS * (A * (A + 1) + 1) + col * A * A + b;
  const Cx<P>* in = T + (size_t)slot * n2 * N1 + c0;
  for (int q = threadIdx.x; q < n2 * COLS; q += TH) tile[q] = in[(size_t)(q / COLS) * N1 + q % COLS];
  __syncthreads();
  Cx<P> x[A];
#pragma unroll
  for (int q = 0; q < A; q++) {
    const int u = q * A + b, jy = a.jy[u];
    x[q] = jy >= 0 ? lerp<P>(tile[jy * COLS + col], tile[(jy + 1) * COLS + col], a.wy[u]) : cx<P>(0, 0);
  }
  fft<P, A, false>(x, tw, buf, b);
  if (SPECTRUM<P>) {
#pragma unroll
    for (int q = 0; q < A; q++) spec[q * A] = x[reversed(q, A)];
  }
  constexpr bool BY_COLUMN = !SPECTRUM<P>;  // the filters' layout
  const size_t h0 = BY_COLUMN ? (size_t)(c0 + col) * N2 + b : (size_t)b * N1 + c0 + col;
  const int hs = BY_COLUMN ? A : A * N1;
#pragma unroll 1
  for (int f = 0; f < 2; f++) {
    const Cx<P>* H = (f ? a.sH2 : a.sH1) + h0;
    Cx<P> y[A];
#pragma unroll
    for (int q = 0; q < A; q++) y[q] = mul<P>(SPECTRUM<P> ? spec[q * A] : x[reversed(q, A)], __ldg(H + hs * q));  // frequency A q + b
    fft<P, A, true>(y, tw, buf, b);
    __syncwarp();
#pragma unroll
    for (int d = 0; d < A; d++) buf[b + A * d] = y[reversed(d, A)];
    __syncthreads();  // (the tile's earlier use is over, too)
    const int rows = n2 + f;
    const int* j2 = f ? a.hy_j2 : a.hx_j2;
    const Re<P>* w2 = f ? a.hy_w2 : a.hx_w2;
    for (int r = b; r < rows; r += A) {
      const int q = j2[r];
      const Cx<P> lo = buf[q], hi = q + 1 < N2 ? buf[q + 1] : cx<P>(0, 0);  // past the last node: zero
      tile[r * COLS + col] = lerp<P>(lo, hi, w2[r]);
    }
    __syncthreads();
    Cx<P>* out = (f ? T2 + (size_t)slot * (n2 + 1) * N1 : T1 + (size_t)slot * n2 * N1) + c0;
    for (int q = threadIdx.x; q < rows * COLS; q += TH) out[(size_t)(q / COLS) * N1 + q % COLS] = tile[q];
  }
}

// rows 0..n2-1: Hx's ghosts from T1, n2..2 n2: Hy's from T2. grid (rows, slots) in groups of A
// lanes. Shared: per group A (A + 1)
template <class P, int A>
__global__ void __launch_bounds__(128) k_air_ghosts(AirP<P> a, const Cx<P>* tw, const Cx<P>* T1, const Cx<P>* T2,
                                                    Cx<P>* ghx, Cx<P>* ghy)
{
  extern __shared__ char raw[];
  Cx<P>* const smem = (Cx<P>*)raw;
  constexpr int G = GROUPS<A>;
  const int grp = threadIdx.x / A, b = threadIdx.x % A;
  const int n1 = a.n1, n2 = a.n2, N1 = a.N1, slot = blockIdx.y;
  const int row = min(blockIdx.x * G + grp, 2 * n2);
  Cx<P>* buf = smem + grp * (A * (A + 1));
  const bool hy = row >= n2;
  const int j = hy ? row - n2 : row;
  const Cx<P>* in = hy ? T2 + ((size_t)slot * (n2 + 1) + j) * N1 : T1 + ((size_t)slot * n2 + j) * N1;
  Cx<P> x[A];
#pragma unroll
  for (int q = 0; q < A; q++) x[q] = in[A * q + b];
  fft<P, A, true>(x, tw, buf, b);
  __syncwarp();
  const Re<P> s = 1 / ((Re<P>)N1 * (Re<P>)a.N2);
#pragma unroll
  for (int d = 0; d < A; d++) {
    const Cx<P> v = x[reversed(d, A)];
    buf[b + A * d] = cx<P>(s * v.x, s * v.y);
  }
  __syncwarp();
  const int n = hy ? n1 : n1 + 1;
  const int* j1 = hy ? a.hy_j1 : a.hx_j1;
  const Re<P>* w1 = hy ? a.hy_w1 : a.hx_w1;
  Cx<P>* out = hy ? ghy + ((size_t)slot * (n2 + 1) + j) * n1 : ghx + ((size_t)slot * n2 + j) * (n1 + 1);
  for (int i = b; i < n; i += A) {
    const int q = j1[i];
    out[i] = lerp<P>(buf[q], q + 1 < N1 ? buf[q + 1] : cx<P>(0, 0), w1[i]);
  }
}

static int side(int N) { return N == 64 ? 8 : (N == 256 ? 16 : (N == 1024 ? 32 : 0)); }
template <class P> static size_t rows_smem(int A, int n1) { return (size_t)(128 / A) * (n1 + A * (A + 1)) * sizeof(Cx<P>); }
template <class P> static size_t columns_smem(int A, int n2)
{
  return (size_t)(COL_THREADS<P> / A) * (n2 + 1 + A * (A + 1) + 1 + (SPECTRUM<P> ? A * A : 0)) * sizeof(Cx<P>);
}

// Square grids: of others the two-dimensional transforms reproduce the reference's, which takes
// n1fft for the slow axis (airbc_init_free.c:48-49 plans n1fft x n2fft; the data is n2fft rows of n1fft).
// Fewer rows than the uniform grid's, so that the buffers are the smaller ones; in complex64 two
// CTAs per SM (complex128: one).
bool air_lines_fit(int n1, int n2, int N1, int N2)
{
  const int A = side(N1);
  return A && N1 == N2 && n2 < N2 && 2 * rows_smem<F32>(A, n1) <= 226 * 1024 && 2 * columns_smem<F32>(A, n2) <= 226 * 1024 &&
         columns_smem<F64>(A, n2) <= SMEM_MOST;
}

std::vector<double2> air_twiddles(int N)
{
  std::vector<double2> t((size_t)N);
  const int A = side(N);
  for (int c = 0; c < A; c++)
    for (int b = 0; b < A; b++) {
      const double th = -2.0 * M_PI * b * c / N;
      t[(size_t)c * A + b] = make_double2(cos(th), sin(th));
    }
  return t;
}

template <class P, int A>
static void launch_air(const GridP<P>& g, const AirP<P>& a, const SysScal<P>* scal, const Cx<P>* X, const int* sys_list,
                       const Cx<P>* tw, Cx<P>* T, Cx<P>* T12, Cx<P>* ghx, Cx<P>* ghy, int nslot,
                       cudaStream_t st)
{
  constexpr int G = GROUPS<A>, TH = COL_THREADS<P>;
  Cx<P> *T1 = T12, *T2 = T12 + (size_t)nslot * a.n2 * a.N1;
  const size_t sr = rows_smem<P>(A, a.n1), sc = columns_smem<P>(A, a.n2), sg = (size_t)G * A * (A + 1) * sizeof(Cx<P>);
  allow_smem<k_air_rows<P, A>>(sr);
  allow_smem<k_air_columns<P, A>>(sc);
  allow_smem<k_air_ghosts<P, A>>(sg);
  count_launch(), k_air_rows<P, A><<<dim3((a.n2 + G - 1) / G, nslot), 128, sr, st>>>(g, a, scal, X, sys_list, tw, T);
  count_launch(), k_air_columns<P, A><<<dim3(a.N1 / (TH / A), nslot), TH, sc, st>>>(a, tw, T, T1, T2);
  count_launch(), k_air_ghosts<P, A><<<dim3((2 * a.n2 + G) / G, nslot), 128, sg, st>>>(a, tw, T1, T2, ghx, ghy);
}

template <class P>
void launch_air_lines(const GridP<P>& g, const AirP<P>& a, const SysScal<P>* scal, const Cx<P>* X, const int* sys_list,
                      const Cx<P>* tw, Cx<P>* T, Cx<P>* T12, Cx<P>* ghx, Cx<P>* ghy, int nslot,
                      cudaStream_t st)
{
  switch (side(a.N1)) {
    case 8: return launch_air<P, 8>(g, a, scal, X, sys_list, tw, T, T12, ghx, ghy, nslot, st);
    case 16: return launch_air<P, 16>(g, a, scal, X, sys_list, tw, T, T12, ghx, ghy, nslot, st);
    default: return launch_air<P, 32>(g, a, scal, X, sys_list, tw, T, T12, ghx, ghy, nslot, st);
  }
}
template void launch_air_lines<F32>(const GridP<F32>&, const AirP<F32>&, const SysScal<F32>*, const float2*, const int*,
                                    const float2*, float2*, float2*, float2*, float2*, int, cudaStream_t);
template void launch_air_lines<F64>(const GridP<F64>&, const AirP<F64>&, const SysScal<F64>*, const double2*, const int*,
                                    const double2*, double2*, double2*, double2*, double2*, int, cudaStream_t);

}  // namespace csem
