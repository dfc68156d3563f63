// y = A x in complex128, the reference's bits (fdfd.c:86-205): the z-marching tiles of
// k_fdfd.cu with the reference's operations in its order.
//
// It is bound by the FP64 unit, 2 operations per SM and cycle. Its 24 quotients per cell,
// 7 FP64 operations each by the / operator, run on the integer units (exact_div.h), and
// products with iwmu and iom, whose real parts are zero, take 2 multiplications: about 60
// FP64 operations per cell instead of 270. Where an operand is out of the quotients' range
// (subnormal, infinite, NaN), or iwmu has a real part, the H value or the output is formed
// again by the / operator.
// 125 x 109 x 93 cells with fvm, three systems in flight: 288 us, 924 us by the / operator.
#include "csem_cuda.cuh"
#include "engine.h"
#include "exact_div.h"

namespace csem {

namespace {

typedef double2 C;

struct Sp {  // a spacing and its reciprocal word
  double d;
  uint64_t R;
};
__device__ __forceinline__ Sp spacing(const double* d, const uint64_t* q, int n)
{
  Sp s;
  s.d = d[n];
  s.R = q ? q[n] : 0;
  return s;
}
// (a - b) / s
__device__ __forceinline__ C dover(C a, C b, Sp s, uint32_t& bad)
{
  return make_double2(xd_div(F64::sub(a.x, b.x), s.d, s.R, bad), xd_div(F64::sub(a.y, b.y), s.d, s.R, bad));
}
// t (i f)
__device__ __forceinline__ C times_i(C t, double f) { return make_double2(-F64::mul(t.y, f), F64::mul(t.x, f)); }

// H at (k, j, i) by the reference's operations (fdfd.c:125-149), zero outside the grid
__device__ __noinline__ void slow_h(const GridP<F64>& g, const C* Ex, const C* Ey, const C* Ez, C iwmu, int k, int j,
                                    int i, C* h)
{
  const int n1 = g.n1, n2 = g.n2, n3 = g.n3, kf = k + g.kstart;
  h[0] = h[1] = h[2] = czero<F64>();
  if (j < n2 && k < n3)
    h[0] = cmul<F64>(csub<F64>(cdivr<F64>(csub<F64>(Ez[ix3(n1, n2, k, j + 1, i)], Ez[ix3(n1, n2, k, j, i)]), g.d2s[j]),
                               cdivr<F64>(csub<F64>(Ey[ix2(n1, n2, k + 1, j, i)], Ey[ix2(n1, n2, k, j, i)]), g.d3s[kf])),
                     iwmu);
  if (i < n1 && k < n3)
    h[1] = cmul<F64>(csub<F64>(cdivr<F64>(csub<F64>(Ex[ix1(n1, n2, k + 1, j, i)], Ex[ix1(n1, n2, k, j, i)]), g.d3s[kf]),
                               cdivr<F64>(csub<F64>(Ez[ix3(n1, n2, k, j, i + 1)], Ez[ix3(n1, n2, k, j, i)]), g.d1s[i])),
                     iwmu);
  if (i < n1 && j < n2)
    h[2] = cmul<F64>(csub<F64>(cdivr<F64>(csub<F64>(Ey[ix2(n1, n2, k, j, i + 1)], Ey[ix2(n1, n2, k, j, i)]), g.d1s[i]),
                               cdivr<F64>(csub<F64>(Ex[ix1(n1, n2, k, j + 1, i)], Ex[ix1(n1, n2, k, j, i)]), g.d2s[j])),
                     iwmu);
}
// an output, ((a - b) / da - (c - d) / dc) - s e, times vol iom with fvm
__device__ __noinline__ C slow_row(C a, C b, double da, C c, C d, double dc, double s, C e, int fvm, double vol, C iom)
{
  C r = csub<F64>(csub<F64>(cdivr<F64>(csub<F64>(a, b), da), cdivr<F64>(csub<F64>(c, d), dc)), rmul<F64>(s, e));
  return fvm ? cmul<F64>(r, rmul<F64>(vol, iom)) : r;
}

}  // namespace

// Threads and tiles as k_fdfd: a warp per j row, a lane per i column, lane 0 and warp 0 the
// halo on the low sides, a chunk of z planes per CTA.
template <int BY>
__global__ void __launch_bounds__(32 * (BY + 1), 1)
k_fdfd64(GridP<F64> g, const SysScal<F64>* __restrict__ scal, const C* __restrict__ X, C* __restrict__ Y,
         const C* __restrict__ GHX, const C* __restrict__ GHY, int kchunk, int nkc, const int* __restrict__ sys_list)
{
  __shared__ C sHx[2][BY + 1][32], sHz[2][BY + 1][32];
  const int lane = threadIdx.x, w = threadIdx.y;
  const int i = blockIdx.x * 31 + lane - 1;
  const int j = blockIdx.y * BY + w - 1;
  const int slot = blockIdx.z / nkc, kc = blockIdx.z % nkc;
  const int sys = sys_list ? sys_list[slot] : slot;
  const int n1 = g.n1, n2 = g.n2, n3 = g.n3, ks = g.kstart;
  const C* Ex = X + (size_t)sys * g.lE;
  const C* Ey = Ex + g.lEx;
  const C* Ez = Ey + g.lEy;
  C* bx = Y + (size_t)sys * g.lE;
  C* by = bx + g.lEx;
  C* bz = by + g.lEy;
  const C iwmu = scal[sys].iwmu, iom = scal[sys].iom;
  const bool fast = g.q1 && iwmu.x == 0. && iom.x == 0.;
  const C* ghx = GHX ? GHX + (size_t)slot * (n1 + 1) * n2 : nullptr;  // ghosts are per slot
  const C* ghy = GHY ? GHY + (size_t)slot * n1 * (n2 + 1) : nullptr;
  const int kb = kc * kchunk, ke = min(n3 + 1, kb + kchunk);
  const bool inside = i >= 0 && j >= 0 && i <= n1 && j <= n2;  // H is zero outside
  const bool interior = lane >= 1 && w >= 1 && inside;         // this thread writes y
  const C z = czero<F64>();
  const bool hasEx = inside && i < n1, hasEy = inside && j < n2, hasExj = hasEx && j < n2;
  const int ic = inside ? i : 0, jc = inside ? j : 0;
  const Sp d1s = spacing(g.d1s, g.q1s, ic), d1 = spacing(g.d1, g.q1, ic);
  const Sp d2s = spacing(g.d2s, g.q2s, jc), d2 = spacing(g.d2, g.q2, jc);
  const bool outX = interior && i < n1, outY = interior && j < n2, outZ = interior;
  const bool inX = j >= 1 && j <= n2 - 1, inY = i >= 1 && i <= n1 - 1, inZ = inX && inY;
  const long sEx = (long)n1 * (n2 + 1), sEy = (long)(n1 + 1) * n2, sEz = (long)(n1 + 1) * (n2 + 1);
  long oEx = inside ? ix1(n1, n2, kb, j, i) : 0;
  long oEy = inside ? ix2(n1, n2, kb, j, i) : 0;
  long oEz = inside ? ix3(n1, n2, kb, j, i) : 0;
  const double* s11 = g.s11 + ks * sEx;
  const double* s22 = g.s22 + ks * sEy;
  const double* s33 = g.s33 + ks * sEz;
  auto Hval = [&](C a, C b, Sp p, C c, C d, Sp q, uint32_t& bad) {
    return times_i(csub<F64>(dover(a, b, p, bad), dover(c, d, q, bad)), iwmu.y);
  };
  auto row = [&](C a, C b, Sp p, C c, C d, Sp q, double s, C e, double va, double vb, double vc) {
    uint32_t bad = fast ? 0u : 1u;
    C r = csub<F64>(csub<F64>(dover(a, b, p, bad), dover(c, d, q, bad)), rmul<F64>(s, e));
    if (g.fvm) r = times_i(r, F64::mul(F64::mul(F64::mul(va, vb), vc), iom.y));
    if (bad) r = slow_row(a, b, p.d, c, d, q.d, s, e, g.fvm, F64::mul(F64::mul(va, vb), vc), iom);
    return r;
  };

  C exk = hasEx ? Ex[oEx] : z;
  C eyk = hasEy ? Ey[oEy] : z;
  C pHx = z, pHy = z;
  if (kb > 0 && inside) {  // Hx and Hy of the plane below the chunk
    uint32_t bad = fast ? 0u : 1u;
    const Sp d3s = spacing(g.d3s, g.q3s, kb - 1 + ks);
    const C ez = Ez[oEz - sEz];
    if (hasEy) pHx = Hval(Ez[oEz - sEz + n1 + 1], ez, d2s, eyk, Ey[oEy - sEy], d3s, bad);
    if (hasEx) pHy = Hval(exk, Ex[oEx - sEx], d3s, Ez[oEz - sEz + 1], ez, d1s, bad);
    if (bad) {
      C h[3];
      slow_h(g, Ex, Ey, Ez, iwmu, kb - 1, j, i, h);
      pHx = h[0];
      pHy = h[1];
    }
  }
  // the loads of one plane: Ez, the j+1 neighbours, Ex and Ey of the plane above, and
  // sigma; issued one plane ahead of their use
  struct PlaneIn {
    C ez, ezj, exj, ex1, ey1;
    double s1, s2, s3;
  };
  auto load_plane = [&](int k, long oX, long oY, long oZ) {
    PlaneIn p;
    const bool kin = k < n3;
    p.ez = inside && kin ? Ez[oZ] : z;
    p.ezj = hasEy && kin ? Ez[oZ + (n1 + 1)] : z;
    p.exj = hasExj ? Ex[oX + n1] : z;
    p.ex1 = hasEx && kin ? Ex[oX + sEx] : z;
    p.ey1 = hasEy && kin ? Ey[oY + sEy] : z;
    p.s1 = outX ? s11[oX] : 0.;
    p.s2 = outY ? s22[oY] : 0.;
    p.s3 = outZ && kin ? s33[oZ] : 0.;
    return p;
  };
  PlaneIn nxt = load_plane(kb, oEx, oEy, oEz);
  for (int k = kb; k < ke; k++, oEx += sEx, oEy += sEy, oEz += sEz) {
    const int kf = k + ks, pb = k & 1;
    const bool kin = k < n3;
    const PlaneIn cur = nxt;
    if (k + 1 < ke) nxt = load_plane(k + 1, oEx + sEx, oEy + sEy, oEz + sEz);
    const Sp d3s = spacing(g.d3s, g.q3s, kf), d3 = spacing(g.d3, g.q3, kf);
    C ezi, eyi;  // Ez(k, j, i+1), Ey(k, j, i+1): the next lane's, loaded by the last lane
    ezi.x = __shfl_down_sync(0xffffffffu, cur.ez.x, 1);
    ezi.y = __shfl_down_sync(0xffffffffu, cur.ez.y, 1);
    eyi.x = __shfl_down_sync(0xffffffffu, eyk.x, 1);
    eyi.y = __shfl_down_sync(0xffffffffu, eyk.y, 1);
    if (lane == 31) {
      ezi = hasEx && kin ? Ez[oEz + 1] : z;
      eyi = hasExj ? Ey[oEy + 1] : z;
    }
    C hx = z, hy = z, hz = z;
    uint32_t bad = fast ? 0u : 1u;
    if (hasEy && kin) hx = Hval(cur.ezj, cur.ez, d2s, cur.ey1, eyk, d3s, bad);
    if (hasEx && kin) hy = Hval(cur.ex1, exk, d3s, ezi, cur.ez, d1s, bad);
    if (hasExj) hz = Hval(eyi, eyk, d1s, cur.exj, exk, d2s, bad);
    if (bad && inside) {
      C h[3];
      slow_h(g, Ex, Ey, Ez, iwmu, k, j, i, h);
      hx = h[0];
      hy = h[1];
      hz = h[2];
    }
    sHx[pb][w][lane] = hx;
    sHz[pb][w][lane] = hz;
    C hyl, hzl;  // Hy(k, j, i-1), Hz(k, j, i-1) from the previous lane
    hyl.x = __shfl_up_sync(0xffffffffu, hy.x, 1);
    hyl.y = __shfl_up_sync(0xffffffffu, hy.y, 1);
    hzl.x = __shfl_up_sync(0xffffffffu, hz.x, 1);
    hzl.y = __shfl_up_sync(0xffffffffu, hz.y, 1);
    __syncthreads();
    if (interior) {
      const C hxd = sHx[pb][w - 1][lane], hzd = sHz[pb][w - 1][lane];  // at j-1
      const bool kxy = (k >= 1 && k <= n3 - 1) || (k == 0 && g.airbc);
      if (outX)
        bx[oEx] = inX && kxy ? row(hz, hzd, d2, hy, k >= 1 ? pHy : ghy[i + (long)n1 * j], d3, cur.s1, exk, d1s.d, d2.d, d3.d)
                             : z;
      if (outY)
        by[oEy] = inY && kxy ? row(hx, k >= 1 ? pHx : ghx[i + (long)(n1 + 1) * j], d3, hz, hzl, d1, cur.s2, eyk, d1.d, d2s.d, d3.d)
                             : z;
      if (outZ && kin) bz[oEz] = inZ ? row(hy, hyl, d1, hx, hxd, d2, cur.s3, cur.ez, d1.d, d2.d, d3s.d) : z;
    }
    pHx = hx;
    pHy = hy;
    exk = cur.ex1;
    eyk = cur.ey1;
  }
}

template <>
void launch_fdfd<F64>(const GridP<F64>& g, const SysScal<F64>* scal, const C* X, C* Y, const C* ghx, const C* ghy,
                      int nsys, const int* sys_list, cudaStream_t st, int by, int ctas_per_sm)
{
  if (by != 4 && by != 16) by = 8;
  const FdfdShape f = fdfd_shape(g.n1, g.n2, g.n3, nsys, by, ctas_per_sm, 31);
  dim3 blk(32, by + 1), grd(f.gx, f.gy, nsys * f.nkc);
  count_launch();
  if (by == 4) k_fdfd64<4><<<grd, blk, 0, st>>>(g, scal, X, Y, ghx, ghy, f.kchunk, f.nkc, sys_list);
  else if (by == 16) k_fdfd64<16><<<grd, blk, 0, st>>>(g, scal, X, Y, ghx, ghy, f.kchunk, f.nkc, sys_list);
  else k_fdfd64<8><<<grd, blk, 0, st>>>(g, scal, X, Y, ghx, ghy, f.kchunk, f.nkc, sys_list);
}

}  // namespace csem
