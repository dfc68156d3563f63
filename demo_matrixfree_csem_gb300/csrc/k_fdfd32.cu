// y = A x in complex64 (fdfd.c:86-205), as the batched solver's inner iterations apply it.
//
// One CTA owns a 30 x BY tile of (i, j) columns and marches a chunk of z planes: a warp per j
// row and a lane per i column, with one more lane on either side and one more row on the low
// side. At each plane a thread forms H = curl E / (i omega mu0) at its column
// (fdfd.c:125-149), trades neighbours (Ey, Ez of the next lane and Hy, Hz of the previous one
// by shuffles, Hx, Hz of the previous row through shared memory, one barrier per plane), and
// y = curl H - sigma E (fdfd.c:176-203). H is never stored.
//
// What bounds it is instruction issue next to memory latency: 28 bytes of DRAM traffic a
// point and component allow about 110 instructions a warp and plane. So nothing in the loop
// is conditional but the stores: columns outside the grid read the nearest one and form
// values that no output takes, as do the extra lanes; the first plane's fields above come as
// the loop's carried values (the airwave's ghosts, fdfd.c:151-172); the last plane of Ex and
// Ey, which only holds zeros, is written apart; and addresses are 32-bit offsets from the
// system's component (64-bit where one has more than 2^29 points, 4 GiB), advanced by one addition
// per component and plane.
// 200 x 140 x 130 cells, 16 systems: 814 us, 3.5 TB/s of DRAM traffic (1049 us with predicated
// loads and 64-bit addresses); tiles 4 and 16 rows high 850 and 1070 us. Of about 230
// instructions a warp and plane 70 are arithmetic; registers (72, for three CTAs of 8 rows
// on an SM) limit the loads in flight.
#include <algorithm>
#include <type_traits>
#include "csem_cuda.cuh"
#include "engine.h"
#include "k_dot_common.cuh"
#include "offsets32.h"

namespace csem {

namespace {

typedef float2 C;

template <class Off> __device__ __forceinline__ C ld(const char* base, Off off) { return __ldg((const C*)(base + off)); }
template <class Off> __device__ __forceinline__ float ldf(const char* base, Off off)
{
  return __ldg((const float*)(base + off));
}
__device__ __forceinline__ C up(C v) { return make_float2(__shfl_up_sync(~0u, v.x, 1), __shfl_up_sync(~0u, v.y, 1)); }
__device__ __forceinline__ C down(C v) { return make_float2(__shfl_down_sync(~0u, v.x, 1), __shfl_down_sync(~0u, v.y, 1)); }
// (roundings written out, so that a value is the same whichever code forms it: the bits do
// not depend on the tile's height or the chunks)
// (a - b) p - (c - d) q
__device__ __forceinline__ float curl(float a, float b, float p, float c, float d, float q)
{
  return __fmaf_rn(__fsub_rn(a, b), p, -__fmul_rn(__fsub_rn(c, d), q));
}
__device__ __forceinline__ C curl(C a, C b, float p, C c, C d, float q)
{
  return make_float2(curl(a.x, b.x, p, c.x, d.x, q), curl(a.y, b.y, p, c.y, d.y, q));
}
__device__ __forceinline__ C mul(C a, C b)
{
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ C less(C a, float s, C b) { return make_float2(__fmaf_rn(-s, b.x, a.x), __fmaf_rn(-s, b.y, a.y)); }

// the values of one plane, loaded a plane ahead: Ez here and at j+1, Ex at j+1, Ex and Ey
// of the plane above, and the conductivities
struct Plane {
  C ez, ezj, exj, ex1, ey1;
  float s1, s2, s3;
};

}  // namespace

// EPI > 0 folds the Krylov dot products of the result into the pass: EPI 1 sums y conj(e)
// (BiCGStab's v.r0 after v = A p), EPI 2 sums e conj(y) and y conj(y) (s.t and t.t after
// t = A s), e read at the outputs' own indices. Each thread accumulates as the dot-product
// kernels do (compensated float pairs), the CTA sums its threads in a fixed tree and order,
// and writes part[slot][cta] (EPI 2: and part[nslot + slot][cta]), which launch_dot_finish
// adds up in a fixed order: deterministic, but a different partition of the sum than
// launch_dot's.
template <int BY, int EPI, class Off>
__global__ void __launch_bounds__(32 * (BY + 1), BY >= 16 ? 1 : (BY >= 8 ? 3 : 5))
    k_fdfd32(GridP<F32> g, const SysScal<F32>* __restrict__ scal, const C* __restrict__ X, C* __restrict__ Y,
             const C* __restrict__ GHX, const C* __restrict__ GHY, int kchunk, int nkc, const int* __restrict__ sys_list,
             const C* __restrict__ E, double2* __restrict__ part)
{
  __shared__ float4 sH[2][BY + 1][32];  // (Hx, Hz) of each row
  const int lane = threadIdx.x, w = threadIdx.y;
  const int i = blockIdx.x * 30 + lane, j = blockIdx.y * BY + w - 1;
  const int slot = blockIdx.z / nkc, kc = blockIdx.z - slot * nkc;
  const int sys = sys_list ? sys_list[slot] : slot;
  const int n1 = g.n1, n2 = g.n2, n3 = g.n3, ks = g.kstart;
  const int kb = kc * kchunk, ke = min(n3, kb + kchunk);  // planes kb..ke-1, and n3 apart
  const size_t so = (size_t)sys * g.lE;
  const char* const Ex = (const char*)(X + so);
  const char* const Ey = (const char*)(X + so + g.lEx);
  const char* const Ez = (const char*)(X + so + g.lEx + g.lEy);
  char* const bx = (char*)(Y + so);
  char* const by = (char*)(Y + so + g.lEx);
  char* const bz = (char*)(Y + so + g.lEx + g.lEy);
  const C iwmu = scal[sys].iwmu, iom = scal[sys].iom;
  const Off sX = 8 * (Off)n1 * (n2 + 1), sY = 8 * (Off)(n1 + 1) * n2, sZ = 8 * (Off)(n1 + 1) * (n2 + 1);  // bytes from plane to plane
  const char* const s11 = (const char*)(g.s11) + (size_t)ks * (sX / 2);
  const char* const s22 = (const char*)(g.s22) + (size_t)ks * (sY / 2);
  const char* const s33 = (const char*)(g.s33) + (size_t)ks * (sZ / 2);
  // the nearest column that each component has
  const int ix = min(i, n1 - 1), iy = min(i, n1), jx = min(max(j, 0), n2), jy = min(jx, n2 - 1);
  // column 0 has no left neighbour that counts and column n1 holds zeros only: both come with the
  // first and the last tile, on the lanes that are else extra
  const bool mine = (lane >= 1 || i == 0) && (lane <= 30 || i == n1) && w >= 1 && i <= n1 && j <= n2;
  const bool outX = mine && i < n1, outY = mine && j < n2, outZ = mine;
  const bool inX = j >= 1 && j <= n2 - 1, inY = i >= 1 && i <= n1 - 1, inZ = inX && inY;
  Off oX = point_offset<Off>(ix, jx, kb, n1, sX), oY = point_offset<Off>(iy, jy, kb, n1 + 1, sY),
      oZ = point_offset<Off>(iy, jx, kb, n1 + 1, sZ);
  const Off upX = jx < n2 ? 8 * (Off)n1 : 0, upZ = jx < n2 ? 8 * (Off)(n1 + 1) : 0;  // to row j + 1
  const float r1s = g.r1s[ix], r1 = g.r1[iy], r2s = g.r2s[jy], r2 = g.r2[jx];
  const float v1s = g.d1s[ix], v1 = g.d1[iy], v2s = g.d2s[jy], v2 = g.d2[jx];
  const C z = make_float2(0.f, 0.f);
  const char* const eX = EPI ? (const char*)(E + so) : nullptr;  // the dot products' other vector
  const char* const eY = EPI ? (const char*)(E + so + g.lEx) : nullptr;
  const char* const eZ = EPI ? (const char*)(E + so + g.lEx + g.lEy) : nullptr;
  DotAcc<F32> dacc1, dacc2;
  auto put = [&](char* out, const char* e, Off o, C y) {
    *(C*)(out + o) = y;
    if constexpr (EPI == 1) {
      dacc1.add(y, ld(e, o));
    } else if constexpr (EPI == 2) {
      dacc1.add(ld(e, o), y);
      dacc2.add(y, y);
    }
  };

  auto load = [&](Off x, Off y, Off zz) {
    Plane p;
    p.ez = ld(Ez, zz);
    p.ezj = ld(Ez, zz + upZ);
    p.exj = ld(Ex, x + upX);
    p.ex1 = ld(Ex, x + sX);
    p.ey1 = ld(Ey, y + sY);
    p.s1 = ldf(s11, x / 2);
    p.s2 = ldf(s22, y / 2);
    p.s3 = ldf(s33, zz / 2);
    return p;
  };
  C pHx = z, pHy = z;  // of the plane below
  if (kb > 0) {
    const C ez = ld(Ez, oZ - sZ), ezi = down(ez);
    const float r3s = g.r3s[kb - 1 + ks];
    pHx = mul(curl(ld(Ez, oZ - sZ + upZ), ez, r2s, ld(Ey, oY), ld(Ey, oY - sY), r3s), iwmu);
    pHy = mul(curl(ld(Ex, oX), ld(Ex, oX - sX), r3s, ezi, ez, r1s), iwmu);
  } else if (GHX) {
    pHx = GHX[(size_t)slot * (n1 + 1) * n2 + iy + (long)(n1 + 1) * jy];
    pHy = GHY[(size_t)slot * n1 * (n2 + 1) + ix + (long)n1 * jx];
  }
  C exk = ld(Ex, oX), eyk = ld(Ey, oY);
  auto plane = [&](int k, const Plane& p, Plane& nxt) {
    const int kf = k + ks;
    if (k + 1 < ke) nxt = load(oX + sX, oY + sY, oZ + sZ);
    const float r3s = g.r3s[kf], r3 = g.r3[kf];
    const C ezi = down(p.ez), eyi = down(eyk);
    const C hx = mul(curl(p.ezj, p.ez, r2s, p.ey1, eyk, r3s), iwmu);
    const C hy = mul(curl(p.ex1, exk, r3s, ezi, p.ez, r1s), iwmu);
    const C hz = mul(curl(eyi, eyk, r1s, p.exj, exk, r2s), iwmu);
    sH[k & 1][w][lane] = make_float4(hx.x, hx.y, hz.x, hz.y);
    const C hyl = up(hy), hzl = up(hz);  // Hy, Hz at i-1
    __syncthreads();
    if (w > 0) {
      const float4 d = sH[k & 1][w - 1][lane];  // Hx, Hz at j-1
      const C hxd = make_float2(d.x, d.y), hzd = make_float2(d.z, d.w);
      C rx = less(curl(hz, hzd, r2, hy, pHy, r3), p.s1, exk);
      C ry = less(curl(hx, pHx, r3, hz, hzl, r1), p.s2, eyk);
      C rz = less(curl(hy, hyl, r1, hx, hxd, r2), p.s3, p.ez);
      if (g.fvm) {
        const float v3s = g.d3s[kf], v3 = g.d3[kf];
        const float fx = v1s * v2 * v3, fy = v1 * v2s * v3, fz = v1 * v2 * v3s;
        rx = mul(rx, make_float2(fx * iom.x, fx * iom.y));
        ry = mul(ry, make_float2(fy * iom.x, fy * iom.y));
        rz = mul(rz, make_float2(fz * iom.x, fz * iom.y));
      }
      const bool kxy = k >= 1 || g.airbc;
      if (outX) put(bx, eX, oX, inX && kxy ? rx : z);
      if (outY) put(by, eY, oY, inY && kxy ? ry : z);
      if (outZ) put(bz, eZ, oZ, inZ ? rz : z);
    }
    pHx = hx;
    pHy = hy;
    exk = p.ex1;
    eyk = p.ey1;
    oX += sX;
    oY += sY;
    oZ += sZ;
  };
  Plane a, b;
  if (kb < ke) a = load(oX, oY, oZ);
  int k = kb;
  for (; k + 1 < ke; k += 2) {
    plane(k, a, b);
    plane(k + 1, b, a);
  }
  if (k < ke) plane(k, a, b);
  if (kb + kchunk > n3) {  // plane n3 of Ex and Ey
    if (outX) put(bx, eX, oX, z);
    if (outY) put(by, eY, oY, z);
  }
  if constexpr (EPI > 0) {
    __shared__ double2 red[2][BY + 1];
    const double2 v1 = warp_sum(dacc1.value());
    const double2 v2 = EPI == 2 ? warp_sum(dacc2.value()) : make_double2(0, 0);
    if (lane == 0) {
      red[0][w] = v1;
      red[1][w] = v2;
    }
    __syncthreads();
    if (w == 0 && lane == 0) {
      double2 a1 = make_double2(0, 0), a2 = make_double2(0, 0);
      for (int q = 0; q <= BY; q++) {
        a1.x = __dadd_rn(a1.x, red[0][q].x);
        a1.y = __dadd_rn(a1.y, red[0][q].y);
        a2.x = __dadd_rn(a2.x, red[1][q].x);
        a2.y = __dadd_rn(a2.y, red[1][q].y);
      }
      const int npart = gridDim.x * gridDim.y * nkc, nslot = gridDim.z / nkc;
      const int cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * kc);
      part[(size_t)slot * npart + cta] = a1;
      if (EPI == 2) part[(size_t)(nslot + slot) * npart + cta] = a2;
    }
  }
}

namespace {

// tiles for columns 1 .. n1 - 1 (a tile more for column 0 or n1 alone made n1 = 30 and 61 slower than
// tiles of 31 did: 30 x 140 x 120 cells, 6 systems, 88 us with those, 105 with the second tile, 67 now)
FdfdShape shape(int n1, int n2, int n3, int nsys, int by, int ctas_per_sm)
{
  return fdfd_shape(std::max(n1 - 2, 0), n2, n3, nsys, by, ctas_per_sm, FDFD32_TILE);
}

template <int EPI>
void launch_by(const GridP<F32>& g, const SysScal<F32>* scal, const C* X, C* Y, const C* ghx, const C* ghy, int nsys,
               const int* sys_list, cudaStream_t st, int by, int ctas_per_sm, const C* E, double2* part)
{
  if (by != 4 && by != 16) by = 8;
  const FdfdShape f = shape(g.n1, g.n2, g.n3, nsys, by, ctas_per_sm);
  dim3 blk(32, by + 1), grd(f.gx, f.gy, nsys * f.nkc);
  auto go = [&](auto tile, auto off) {
    constexpr int BY = decltype(tile)::value;
    typedef decltype(off) Off;
    // of 228 KB; three CTAs use 28 (16 systems' operators on three streams: 1094 -> 921 us each)
    keep_l1<k_fdfd32<BY, EPI, Off>>(20);
    count_launch(), k_fdfd32<BY, EPI, Off><<<grd, blk, 0, st>>>(g, scal, X, Y, ghx, ghy, f.kchunk, f.nkc, sys_list, E, part);
  };
  auto with = [&](auto off) {
    if (by == 4) go(std::integral_constant<int, 4>(), off);
    else if (by == 16) go(std::integral_constant<int, 16>(), off);
    else go(std::integral_constant<int, 8>(), off);
  };
  if (offsets32_reach(g.n1, g.n2, g.n3)) with(0u);
  else with((size_t)0);
}

}  // namespace

template <>
void launch_fdfd<F32>(const GridP<F32>& g, const SysScal<F32>* scal, const C* X, C* Y, const C* ghx, const C* ghy,
                      int nsys, const int* sys_list, cudaStream_t st, int by, int ctas_per_sm)
{
  launch_by<0>(g, scal, X, Y, ghx, ghy, nsys, sys_list, st, by, ctas_per_sm, nullptr, nullptr);
}

void launch_fdfd_dot(const GridP<F32>& g, const SysScal<F32>* scal, const float2* X, float2* Y, const float2* ghx,
                     const float2* ghy, int nsys, const int* sys_list, cudaStream_t st, int by, int ctas_per_sm,
                     int kind, const float2* E, double2* part)
{
  if (kind == 2) launch_by<2>(g, scal, X, Y, ghx, ghy, nsys, sys_list, st, by, ctas_per_sm, E, part);
  else launch_by<1>(g, scal, X, Y, ghx, ghy, nsys, sys_list, st, by, ctas_per_sm, E, part);
}

int fdfd_partials(int n1, int n2, int n3, int nsys, int by, int ctas_per_sm)
{
  const FdfdShape f = shape(n1, n2, n3, nsys, by, ctas_per_sm);
  return f.gx * f.gy * f.nkc;
}

}  // namespace csem
