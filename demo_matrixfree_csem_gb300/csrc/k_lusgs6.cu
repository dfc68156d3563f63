// complex64 LU-SGS component sweeps as a pass over all points and a chain with a warp per line.
//
// A component sweep in linear form (k_sweep_common.cuh) is v(r, m) = B + w (gp v(r, m-1) +
// gn v(r-1, m)) going forward, the upper neighbours going backward, on independent lines:
// Ex rows k, march j, lines i; Ey rows k, march i, lines j; Ez rows j, march i, lines k. B and
// w hold only what nothing writes during the sweep before the point is reached. So a pass
// (k_line_pass, k_line_pass_ex) stores B of every point, and w once for the systems of a
// frequency, in the order in which the chain works through a line (line_entry). What is left
// for the chain (k_line32) is two 8-byte loads, six multiply-adds and an 8-byte store per
// point, and the dependence.
//
// The pass: a thread per point, which forms 1/aii and w once for its frequency's systems. A
// point's operands lie at the same offsets in every system, so they are formed once, too,
// relative to the planes k and k-1 (k+1 for Ez), each in y or in the cap. Ex's lines are
// i, the axis its operands are contiguous on, so 32 x 16 tiles turn in shared memory. A thread
// forms two points, for the loads in flight; Ey's and Ez's are of neighbouring rows j and share
// some (11 -> 9 or 10 a point). 64 registers (Ex 80), for 32 warps an SM (24).
//
// The chain: a warp owns one line and works through its march in strips of 32 positions, lane t on
// position t of the strip, over all rows of the strip before the next strip. Lane t runs t
// rows behind lane 0, so that lane t - 1's value at its row is there, one shuffle away, when
// it is due. Loads and stores stay together all the same: rows are copied into a queue in
// shared memory (cp.async, 9 to 16 rows early), where lane t takes its entry t steps after
// lane 0 and leaves v in its place; 31 steps after lane 0 the row is complete and is stored by
// all lanes at once. A strip's last column is kept for the left neighbours
// of the next strip's first (edge), and the strips follow one another without draining:
// lanes go over to the next strip one by one. Everything that does not happen at every row
// happens every 8 rows (4 in some shapes, launch_line), and the copies and stores are a second
// warp's, one barrier a chunk apart from the first: with one or two lines' warps to a scheduler
// every instruction counts towards the line's time, and a chunk's 8 rows took 700 cycles of the
// chain and 550 of the rest in turn.
//
// Ex is the contiguous axis across its lines: a CTA takes 8 (or 4) neighbouring lines and stores
// their rows together, 64 bytes at a time.
//
// The thread-per-row pipelines (k_sweep_ex32s, k_sweep_eyz32s, lusgs_split 1) read one 16-byte
// entry per row and lane, 20 sectors a request, and join a line's warps by barriers at every
// step. Per application, them, this with one warp to a line and one point to a pass's thread, and
// this, one context: 200 x 140 x 140 cells, 48 systems 23.3, 14.6, 12.8 ms, 16 systems 8.02,
// 5.30, 4.42, 3 systems 2.11, 1.40, 1.07; 84^3 cells, 6 systems 0.86, 0.51, 0.39; 81 x 73 x 67
// cells, 3 systems at 3 frequencies 0.51, 0.35, 0.25. The pass takes 60% of it, at 60% of the
// DRAM rate, bound by its loads' latency; the chain runs at 50% (large batches: 7 or 8 lines on
// an SM by its shared memory, and its load and store unit) or is bound by its steps' latency, 640
// cycles for 8 rows (small ones).
#include <algorithm>
#include <type_traits>
#include "csem_cuda.cuh"
#include "engine.h"
#include "k_sweep_common.cuh"

namespace csem {

using namespace sweep;

namespace {

typedef float2 C;

__device__ __forceinline__ void fetch16(unsigned dst, const void* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A CTA's lines (Ey, Ez: 1; Ex: 4 or 8), rows per chunk (8 or 4), chunks copied ahead
template <int LINES, int CH> struct LineShape {
  static constexpr int AHEAD = CH == 4 ? 3 : 2;
  static constexpr int DEPTH = 32 + CH * (1 + AHEAD);  // queue entries per lane: 32 rows in work or to be stored, and the copies
  // a line's queue in float2: B (and then v) [DEPTH][32], w [DEPTH][32], padding (Ex's lines on
  // different banks)
  static constexpr int QUEUE = 2 * DEPTH * 32 + (LINES > 1 ? 16 / LINES : 0);
};
constexpr unsigned QE = 256;  // bytes from a lane's queue entry to its next

// shared memory: queues, edge columns float2 [warps][Rp + 32], row couplings float [32 + Rp]
// (the first 32: the last rows of the strip before)
template <int LINES, int CH> inline size_t line_smem(int R)
{
  const size_t Rp = line_steps(R);
  return LINES * (LineShape<LINES, CH>::QUEUE * 8 + (Rp + 32) * 8) + (Rp + 32) * 4;
}

// A point's coupling to the other two components and its own not-yet-swept neighbours, at
// offsets (in bytes) that all systems share: from plane k's memory (A) and from the second
// plane's (B: k-1, for Ez k+1)
__device__ __forceinline__ C at(const char* base, unsigned off) { return ro((const C*)(base + off)); }

// A group's slots and systems, one member per lane (in the first lanes)
template <int NS> struct Members {
  int slot, sys, n;
  __device__ __forceinline__ Members(const SweepP<F32>& s, const int* groups, int grp)
  {
    const int lane = threadIdx.x & 31;
    slot = NS > 1 ? (lane < NS ? groups[(size_t)grp * NS + lane] : -1) : grp;
    sys = slot < 0 ? 0 : (s.sys_list ? s.sys_list[slot] : slot);
    n = NS > 1 ? __popc(__ballot_sync(0xffffffffu, slot >= 0)) : 1;
  }
  __device__ __forceinline__ int slot_of(int q) const { return NS > 1 ? __shfl_sync(0xffffffffu, slot, q) : slot; }
  __device__ __forceinline__ int sys_of(int q) const { return NS > 1 ? __shfl_sync(0xffffffffu, sys, q) : sys; }
};
// Per-system bases of the two planes
struct Bases {
  const char *A, *B, *x;
};
__device__ __forceinline__ Bases bases(const SweepP<F32>& s, int slot, int sys, bool upA, bool upB)
{
  const char* y = (const char*)(s.Y + (size_t)sys * s.g.lE);
  const char* c = (const char*)(s.CAP + (size_t)slot * s.capE);
  Bases b;
  b.A = upA ? y : c;
  b.B = upB ? y : c;
  b.x = (const char*)(s.X + (size_t)sys * s.g.lE);
  return b;
}
// offset of component c's plane k in its memory
__device__ __forceinline__ long plane(const SweepP<F32>& s, int c, int k, bool up)
{
  const GridP<F32>& g = s.g;
  const long kk = up ? k - s.vshift : k;
  if (c == 0) return kk * g.n1 * (g.n2 + 1);
  if (c == 1) return (up ? g.lEx : s.capEx) + kk * (g.n1 + 1) * g.n2;
  return (up ? g.lEx + g.lEy : s.capEx + s.capEy) + kk * (g.n1 + 1) * (g.n2 + 1);
}

// 1 / (a + i low) as v + c, good to some 2^-40: scaled, so that no square leaves the range, and a step
// of Newton's iteration from the residual, whose products are formed exactly
struct Recip {
  C v, c;
};
__device__ __forceinline__ float rcp_approx(float a)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ Recip recip(C a, float low)
{
  const float rm = rcp_approx(fmaxf(fabsf(a.x), fabsf(a.y)));
  const float xs = a.x * rm, ys = a.y * rm, q = rm * rcp_approx(__fmaf_rn(xs, xs, ys * ys));
  const float x = xs * q, y = -ys * q;
  const float h = __fmul_rn(a.x, x), k = -__fmul_rn(a.y, y), m = __fmul_rn(a.y, x);  // h + k is 1, nearly
  const float hl = __fmaf_rn(a.x, x, -h), kl = -__fmaf_rn(a.y, y, k), ml = __fmaf_rn(a.y, x, -m);
  const float er = __fsub_rn(__fsub_rn(__fsub_rn(1.f, fmaxf(h, k)), fminf(h, k)), __fsub_rn(__fadd_rn(hl, kl), low * y));
  const float ei = -__fadd_rn(__fmaf_rn(a.x, y, m), __fmaf_rn(low, x, ml));
  Recip r;
  r.v = make_float2(x, y);
  r.c = make_float2(__fmaf_rn(x, er, -__fmul_rn(y, ei)), __fmaf_rn(x, ei, __fmul_rn(y, er)));
  return r;
}
// What a point and a frequency share: w = iwmu/aii with aii = (ga + gb) iwmu - sg, and 1/aii (with
// fvm 1/(aii vol iom)), both to the last place of aii from the rounded reciprocal spacings: their
// errors are the same all along a line, and add up. Of 41 A-phi models the output's error is
// 0.996 times that of the sweeps by diagonals, which divide (1.025, and up to 1.7, with 1/aii and w
// of some three places' error), of 16 LU-SGS models 0.60 times that of the row pipelines
struct Coef {
  C inv, w;
};
__device__ __forceinline__ Coef coef(const SysScal<F32>& sc, int fvm, float2 ga, float2 gb, float sg, float vol)
{
  const float g = __fadd_rn(ga.x, gb.x), t = __fsub_rn(g, ga.x);
  const float gl = __fadd_rn(__fadd_rn(__fsub_rn(ga.x, __fsub_rn(g, t)), __fsub_rn(gb.x, t)), __fadd_rn(ga.y, gb.y));
  const C iw = sc.iwmu;
  const float y = __fmul_rn(g, iw.y), yl = __fmaf_rn(gl, iw.y, __fmaf_rn(g, iw.y, -y));
  const Recip r = recip(make_float2(__fmaf_rn(g, iw.x, -sg), y), yl);
  Coef c;
  c.inv = make_float2(__fadd_rn(r.v.x, r.c.x), __fadd_rn(r.v.y, r.c.y));
  c.w.x = __fmaf_rn(iw.x, r.v.x, __fmaf_rn(-iw.y, r.v.y, __fmaf_rn(iw.x, r.c.x, -__fmul_rn(iw.y, r.c.y))));
  c.w.y = __fmaf_rn(iw.y, r.v.x, __fmaf_rn(iw.x, r.v.y, __fmaf_rn(iw.y, r.c.x, __fmul_rn(iw.x, r.c.y))));
  if (fvm) {
    const Recip f = recip(make_float2(vol * sc.iom.x, vol * sc.iom.y), 0.f);
    c.inv = mul32(c.inv, make_float2(__fadd_rn(f.v.x, f.c.x), __fadd_rn(f.v.y, f.c.y)));
  }
  return c;
}
// B = b/aii + w kc (with fvm b/(aii vol iom)), kc = known - cross
__device__ __forceinline__ C form_B(const Coef& c, C b, C kc)
{
  return make_float2(__fmaf_rn(b.x, c.inv.x, __fmaf_rn(-b.y, c.inv.y, __fmaf_rn(c.w.x, kc.x, -__fmul_rn(c.w.y, kc.y)))),
                     __fmaf_rn(b.x, c.inv.y, __fmaf_rn(b.y, c.inv.x, __fmaf_rn(c.w.x, kc.y, __fmul_rn(c.w.y, kc.x)))));
}

constexpr int PASS_WARPS = 2;
// Percent of an SM's 228 KB that the passes leave for shared memory (Ex's uses 26 KB). With the
// chains' setting (all of it) the passes' loads miss L1: 16 systems 5.80 ms an application instead
// of 4.42, and 5.53 instead of 4.25 where three contexts' applications overlap
constexpr int PASS_SMEM = 20;

}  // namespace

// Ey and Ez: a warp per strip of a pair of rows j, PASS_WARPS pairs. grid (strips x groups, pairs, k)
template <int COMP, bool FWD, int NS>
__global__ void __launch_bounds__(32 * PASS_WARPS, 16)
    k_line_pass(SweepP<F32> s, float2* SB, float2* SW, long sbs, const int* groups)
{
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK, L1 = n1 + 1;
  const int M = n1 - 1, R = COMP == 1 ? nK - 1 : n2 - 1, S = line_strips(M), Rp = line_steps(R);
  const int grp = blockIdx.x / S, strip = blockIdx.x - grp * S;
  const int lane = threadIdx.x & 31, j0 = 2 * (blockIdx.y * PASS_WARPS + (threadIdx.x >> 5)) + (COMP == 2 ? 1 : 0);
  const int k = blockIdx.z + (COMP == 1 ? 1 : 0);
  const int p = strip * 32 + lane, i = FWD ? min(1 + p, M) : max(M - p, 1);
  const Members<NS> mem(s, groups, grp);
  const SysScal<F32> sc = s.scal[mem.sys_of(0)];
  if (j0 >= n2) return;
  // lanes past the last position form position M again, and a last row without a pair is formed
  // twice; neither is stored
  const bool on = p < M, pair = j0 + 1 < n2;
  // Ey: row axis Z (k), line axis Y (j); Ez: row axis Y (j), line axis Z (k)
  const Ax<F32> X = axis<F32>(g.d1, g.d1s, g.r1, g.r1s, i);
  const float2 gx = ro(g.gg1 + i);
  Coef cf[2];
  float rr[2], lrs[2], kr[2];  // the row's 1/d, the line's 1/ds, the coupling to the row below
  size_t e[2];
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const int j = min(j0 + a, n2 - 1);
    const Ax<F32> Rw = COMP == 1 ? axis<F32>(g.d3, g.d3s, g.r3, g.r3s, k) : axis<F32>(g.d2, g.d2s, g.r2, g.r2s, j);
    const Ax<F32> LA = COMP == 1 ? axis_at<F32>(g.d2, g.d2s, g.r2, g.r2s, j) : axis_at<F32>(g.d3, g.d3s, g.r3, g.r3s, k);
    const float2 gr = COMP == 1 ? ro(g.gg3 + k) : ro(g.gg2 + j);  // the row axis' part of aii
    const float ydd = COMP == 1 ? LA.d : Rw.d, zdd = COMP == 1 ? Rw.d : LA.d;
    const float sg = ro(COMP == 1 ? g.s22 + ix2(n1, n2, k, j, i) : g.s33 + ix3(n1, n2, k, j, i));
    cf[a] = coef(sc, g.fvm, gx, gr, sg, X.ds * ydd * zdd);
    rr[a] = Rw.r;
    lrs[a] = -LA.rs;
    kr[a] = Rw.r * Rw.rsm;
    e[a] = line_entry(S, Rp, COMP == 1 ? j : k, p, COMP == 1 ? (FWD ? k - 1 : R - k) : (FWD ? j - 1 : R - j));
    if (on && (a == 0 || pair)) SW[(size_t)grp * sbs + e[a]] = cf[a].w;
  }
  const int kB = COMP == 1 ? k - 1 : k + 1;
  const bool upA = k >= s.vshift, upB = kB >= s.vshift;
  // rows of Ex: Ey j0, j0 + 1, j0 + 2 of plane k; Ez j0, j0 + 1 of planes k and kB. Rows of the
  // third component, both planes: Ey's Ez j0, j0 + 1, j0 + 2; Ez's Ey j0 - 1, j0, j0 + 1
  unsigned xo[4], yo[6], own[2], low[2];
  const unsigned px = 8u * (unsigned)(plane(s, 0, k, upA) + i), py = 8u * (unsigned)(plane(s, 3 - COMP, k, upA) + i);
  const unsigned qy = 8u * (unsigned)(plane(s, 3 - COMP, kB, upB) + i), po = 8u * (unsigned)(plane(s, COMP, k, upA) + i);
  if (COMP == 1) {
    const unsigned ql = 8u * (unsigned)(plane(s, 1, kB, upB) + i);
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const unsigned j = min(j0 + r, n2);
      xo[r] = px + 8u * n1 * j;
      yo[r] = py + 8u * L1 * j;
      yo[3 + r] = qy + 8u * L1 * j;
    }
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const unsigned j = min(j0 + a, n2 - 1);
      own[a] = po + 8u * L1 * j;
      low[a] = ql + 8u * L1 * j;
    }
  } else {
    const unsigned qx = 8u * (unsigned)(plane(s, 0, kB, upB) + i);
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const unsigned j = min(j0 + a, n2 - 1);
      xo[a] = qx + 8u * n1 * j;
      xo[2 + a] = px + 8u * n1 * j;
      own[a] = po + 8u * L1 * j;
      low[a] = own[a] - 8u * L1;
    }
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const unsigned j = min(j0 + r, n2) - 1;
      yo[r] = py + 8u * L1 * j;
      yo[3 + r] = qy + 8u * L1 * j;
    }
  }
  const float km = X.r * X.rsm;
  const C z = make_float2(0.f, 0.f);
  struct Vals {
    C b[2], x[4], xm[4], y[6], o[2], lo[2];
  };
  auto load = [&](int q) {
    const Bases m = bases(s, mem.slot_of(q), mem.sys_of(q), upA, upB);
    Vals v;
#pragma unroll
    for (int a = 0; a < 2; a++) v.b[a] = upA ? at(m.x, own[a]) : z;
#pragma unroll
    for (int r = 0; r < (COMP == 1 ? 3 : 4); r++) {
      const char* const x = COMP == 2 && r < 2 ? m.B : m.A;
      v.x[r] = at(x, xo[r]), v.xm[r] = at(x, xo[r] - 8);
    }
    if (COMP == 2 || !FWD) {
#pragma unroll
      for (int r = 0; r < 6; r++) v.y[r] = at(r < 3 ? m.A : m.B, yo[r]);
    }
    if (!FWD) {
#pragma unroll
      for (int a = 0; a < 2; a++) v.o[a] = at(m.A, own[a] - 8), v.lo[a] = at(COMP == 1 ? m.B : m.A, low[a]);
    }
    return v;
  };
  auto form = [&](int q, const Vals& v) {
    float2* const out = SB + (size_t)mem.slot_of(q) * sbs;
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const int u = COMP == 1 ? a + 1 : a, l = COMP == 1 ? a : a + 2;  // Ex on the upper and the lower side
      const C dx = sub32(sub32(v.x[u], v.x[l]), sub32(v.xm[u], v.xm[l]));
      // Ey: Y.rs (Z.r dEz + X.r dEx); Ez: Z.rs (X.r dEx + Y.r dEy)
      C acc = scl32(X.r, dx);
      if (COMP == 2 || !FWD) {
        const C dy = COMP == 1 ? sub32(sub32(v.y[a + 1], v.y[a]), sub32(v.y[a + 4], v.y[a + 3]))
                               : sub32(sub32(v.y[a + 4], v.y[a + 1]), sub32(v.y[a + 3], v.y[a]));
        acc = make_float2(acc.x + rr[a] * dy.x, acc.y + rr[a] * dy.y);
      }
      C kc = scl32(lrs[a], acc);
      if (!FWD) kc = make_float2(kc.x + (km * v.o[a].x + kr[a] * v.lo[a].x), kc.y + (km * v.o[a].y + kr[a] * v.lo[a].y));
      const C B = form_B(cf[a], v.b[a], kc);
      if (on && (a == 0 || pair)) out[e[a]] = B;
    }
  };
#pragma unroll 1
  for (int q = 0; q < mem.n; q++) form(q, load(q));
}

// Ex: a CTA forms 32 i x half a strip's 16 positions j, along i, and stores them along j, 128 bytes
// a line. 3 CTAs with 80 registers: a barrier per system stops a third of an SM (an application, 48
// systems of 200 x 140 x 140 cells: 12.78 ms; 2 CTAs of whole strips, 64 registers and spills,
// 12.92; 4 of half strips 12.85, 5 13.63). grid (i tiles x groups, half strips, k)
template <bool FWD, int NS>
__global__ void __launch_bounds__(256, 3) k_line_pass_ex(SweepP<F32> s, float2* SB, float2* SW, long sbs, int nti, const int* groups)
{
  __shared__ C tiles[2][32][17];  // one is written while the other's values go out
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, L1 = n1 + 1;
  const int grp = blockIdx.x / nti, i0 = (blockIdx.x - grp * nti) * 32, k = 1 + blockIdx.z;
  const int R = s.nK - 1, M = n2 - 1, S = line_strips(M), Rp = line_steps(R);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int i = min(i0 + tx, n1 - 1);  // (threads past the last line form it again)
  const Members<NS> mem(s, groups, grp);
  const SysScal<F32> sc = s.scal[mem.sys_of(0)];
  const bool upA = k >= s.vshift, upB = k - 1 >= s.vshift;
  const Ax<F32> Z = axis<F32>(g.d3, g.d3s, g.r3, g.r3s, k);
  const float xrs = ro(g.r1s + i), xds = ro(g.d1s + i), kz = Z.r * Z.rsm;
  const float2 gz = ro(g.gg3 + k);
  Coef cf[2];
  float yr[2], kj[2];
  unsigned ox[2], oy[2], oz[2], ozm[2], oxm[2];
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const int st = 16 * blockIdx.y + ty + 8 * a, j = FWD ? min(1 + st, M) : max(M - st, 1);  // (past the last position: it again)
    const Ax<F32> Y = axis<F32>(g.d2, g.d2s, g.r2, g.r2s, j);
    cf[a] = coef(sc, g.fvm, ro(g.gg2 + j), gz, ro(g.s11 + ix1(n1, n2, k, j, i)), xds * Y.d * Z.d);
    yr[a] = Y.r;
    kj[a] = Y.r * Y.rsm;
    ox[a] = 8u * (unsigned)(plane(s, 0, k, upA) + (long)j * n1 + i);
    oxm[a] = 8u * (unsigned)(plane(s, 0, k - 1, upB) + (long)j * n1 + i);
    oy[a] = 8u * (unsigned)(plane(s, 1, k, upA) + (long)j * L1 + i);
    oz[a] = 8u * (unsigned)(plane(s, 2, k, upA) + (long)j * L1 + i);
    ozm[a] = 8u * (unsigned)(plane(s, 2, k - 1, upB) + (long)j * L1 + i);
    tiles[1][tx][ty + 8 * a] = cf[a].w;
  }
  const int sp = threadIdx.x & 15, sl = threadIdx.x >> 4;
  const size_t e0 = line_entry(S, Rp, i0 + sl, 16 * blockIdx.y + sp, FWD ? k - 1 : R - k), e1 = line_entry(S, Rp, 16, 0, 0);
  const bool w0 = i0 + sl < n1, w1 = i0 + sl + 16 < n1;
  auto turn = [&](C(*tile)[17], C* out) {
    __syncthreads();
    if (w0) out[e0] = tile[sl][sp];
    if (w1) out[e0 + e1] = tile[sl + 16][sp];
  };
  turn(tiles[1], SW + (size_t)grp * sbs);
  const C z = make_float2(0.f, 0.f);
  struct Vals {
    C b, ya, yb, yc, yd, za, zb, zc, zd, ej, ek;
  };
  Vals v[2];
  auto load = [&](int q) {
    const Bases m = bases(s, mem.slot_of(q), mem.sys_of(q), upA, upB);
#pragma unroll
    for (int a = 0; a < 2; a++) {
      v[a].b = upA ? at(m.x, ox[a]) : z;
      if (!FWD) {
        const unsigned oyl = oy[a] - 8u * L1;
        v[a].ya = at(m.A, oy[a] + 8), v[a].yb = at(m.A, oy[a]), v[a].yc = at(m.A, oyl + 8), v[a].yd = at(m.A, oyl);
        v[a].za = at(m.A, oz[a] + 8), v[a].zb = at(m.A, oz[a]), v[a].zc = at(m.B, ozm[a] + 8), v[a].zd = at(m.B, ozm[a]);
        v[a].ej = at(m.A, ox[a] - 8u * n1), v[a].ek = at(m.B, oxm[a]);
      }
    }
  };
  load(0);
#pragma unroll 1
  for (int q = 0; q < mem.n; q++) {
    C(*tile)[17] = tiles[q & 1];
#pragma unroll
    for (int a = 0; a < 2; a++) {
      C kc = z;
      if (!FWD) {
        const C dy = sub32(sub32(v[a].ya, v[a].yb), sub32(v[a].yc, v[a].yd));
        const C dz = sub32(sub32(v[a].za, v[a].zb), sub32(v[a].zc, v[a].zd));
        const C cross = scl32(xrs, make_float2(yr[a] * dy.x + Z.r * dz.x, yr[a] * dy.y + Z.r * dz.y));
        kc = sub32(make_float2(kj[a] * v[a].ej.x + kz * v[a].ek.x, kj[a] * v[a].ej.y + kz * v[a].ek.y), cross);
      }
      tile[tx][ty + 8 * a] = form_B(cf[a], v[a].b, kc);
    }
    if (q + 1 < mem.n) load(q + 1);  // in flight while this system's tile turns
    turn(tile, SB + (size_t)mem.slot_of(q) * sbs);
  }
}

// The entries that the sweeps read and never write, the boundary edges, set to zero: planes 0 and
// nK of Ex and Ey, rows j = 0 and n2 of Ex and Ez, columns i = 0 and n1 of Ey and Ez. A tenth of
// clearing all of y (16 systems of 3.7 M points, 1.4 GB: 210 -> 20 us). grid (planes, components,
// slots)
__global__ void __launch_bounds__(128) k_line_bounds(SweepP<F32> s)
{
  const int n1 = s.g.n1, n2 = s.g.n2, L1 = n1 + 1, k = blockIdx.x, c = blockIdx.y, slot = blockIdx.z;
  if (c == 2 && k == s.nK) return;
  const bool up = k >= s.vshift;
  C* const p = (up ? s.Y + (size_t)(s.sys_list ? s.sys_list[slot] : slot) * s.g.lE : s.CAP + (size_t)slot * s.capE) +
               plane(s, c, k, up);
  const int W = c == 0 ? n1 : L1, H = c == 1 ? n2 : n2 + 1;  // a plane's columns and rows
  const C z = make_float2(0.f, 0.f);
  if (c < 2 && (k == 0 || k == s.nK)) {
    for (int q = threadIdx.x; q < W * H; q += 128) p[q] = z;
    return;
  }
  if (c != 1)
    for (int q = threadIdx.x; q < W; q += 128) p[q] = p[(long)(H - 1) * W + q] = z;
  if (c != 0)
    for (int q = threadIdx.x; q < H; q += 128) p[(long)q * W] = p[(long)q * W + n1] = z;
}

// A-phi's backward edge sweeps as LU-SGS's: their extra term, sigma grad v (fdfd.c:735-790, times
// the cell's volume and i omega in finite volumes), goes into the right-hand side T, [slot's
// system][lE]. grid (edges, slots)
__global__ void __launch_bounds__(256) k_aphi_rhs(SweepP<F32> s, C* T)
{
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, n3 = g.n3, L1 = n1 + 1, slot = blockIdx.y;
  const long q = (long)blockIdx.x * 256 + threadIdx.x;
  if (q >= g.lE) return;
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  const C* v = s.V + (size_t)slot * s.lv;
  const int c = q < g.lEx ? 0 : (q < g.lEx + g.lEy ? 1 : 2);
  const unsigned r = (unsigned)(q - (c == 0 ? 0 : (c == 1 ? g.lEx : g.lEx + g.lEy)));
  const unsigned W = c == 0 ? n1 : L1, H = c == 1 ? n2 : n2 + 1;
  const int i = r % W, j = r / W % H, k = r / (W * H);
  C t = ro(s.X + (size_t)sys * g.lE + q);
  if ((c == 0 || (i >= 1 && i < n1)) && (c == 1 || (j >= 1 && j < n2)) && (c == 2 || (k >= 1 && k < n3))) {
    const long n = ix3(n1, n2, k, j, i);
    const C hi = ro(v + n + (c == 0 ? 1 : (c == 1 ? L1 : (long)L1 * (n2 + 1)))), lo = ro(v + n);
    const float f = (c == 0 ? ro(g.s11 + r) * ro(g.r1s + i) : (c == 1 ? ro(g.s22 + r) * ro(g.r2s + j) : ro(g.s33 + r) * ro(g.r3s + k)));
    const C d = sub32(hi, lo);
    if (g.fvm) {
      const SysScal<F32> sc = s.scal[sys];
      const C e = mul32(scl32(f, d), scl32(ro(g.d1s + i) * ro(g.d2 + j) * ro(g.d3 + k), sc.iom));
      t = make_float2(t.x + e.x, t.y + e.y);
    } else {
      t = make_float2(__fmaf_rn(f, d.x, t.x), __fmaf_rn(f, d.y, t.y));
    }
  }
  T[(size_t)sys * g.lE + q] = t;
}

template <int COMP, bool FWD, int LINES, int CH>
__global__ void __launch_bounds__(64 * LINES) k_line32(SweepP<F32> s, const float2* SB, const float2* SW,
                                                                        long sbs, const int* group_of, int groups_per_slot)
{
  typedef LineShape<LINES, CH> Shape;
  constexpr int AHEAD = Shape::AHEAD, DEPTH = Shape::DEPTH, QUEUE = Shape::QUEUE;
  constexpr unsigned QW = DEPTH * QE;  // bytes from a B to its w
  extern __shared__ float2 smem[];
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK;
  const int nlines = COMP == 0 ? n1 : (COMP == 1 ? n2 : nK);
  const int R = COMP == 2 ? n2 - 1 : nK - 1;  // rows 1..R
  const int M = COMP == 0 ? n2 - 1 : n1 - 1;  // march positions 1..M
  const int Rp = line_steps(R);
  const int S = (M + 31) / 32;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % LINES;
  const bool mover = threadIdx.x >= 32 * LINES;  // a line's second warp: its copies and stores
  const int slot = blockIdx.x / groups_per_slot;
  const int line0 = (blockIdx.x - slot * groups_per_slot) * LINES;
  const int line = LINES > 1 ? min(line0 + warp, nlines - 1) : line0;  // (a CTA's warps stay together)
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  const View<F32> V = view_of<F32>(s, slot, sys);
  const C z = make_float2(0.f, 0.f);
  const int L1 = n1 + 1;
  auto row_of = [&](int rho) { return FWD ? 1 + rho : R - rho; };
  auto col = [&](int st) { return FWD ? 1 + 32 * st + lane : M - 32 * st - lane; };

  C* const edge = smem + LINES * QUEUE + warp * (Rp + 32);
  float* const rowgn = (float*)(smem + LINES * QUEUE + LINES * (Rp + 32));
  // what couples a step's row to the row before
  for (int q = threadIdx.x; q < 32 + Rp; q += 64 * LINES) {
    const int rho = q < 32 ? q - 32 + Rp : q - 32;
    float gn = 0.f;
    if (rho < R) {
      const int r = row_of(rho), d = FWD ? r - 1 : r;
      gn = COMP == 2 ? ro(g.r2 + r) * ro(g.r2s + d) : ro(g.r3 + r) * ro(g.r3s + d);
    }
    rowgn[q] = gn;
  }
  for (int q = lane; q < Rp + 32; q += 32) edge[q] = z;

  char* const queue = (char*)(smem + warp * QUEUE + lane);

  // ---- copies: the line's stream of rows of 32 entries, 16 bytes a lane and copy
  const size_t stream = line_entry(S, Rp, line, 0, 0) + 2 * lane;
  const C* sB = SB + (size_t)slot * sbs + stream;
  const C* sW = SW + (size_t)(group_of ? group_of[slot] : slot) * sbs + stream;
  const unsigned queue_a = (unsigned)__cvta_generic_to_shared(smem + warp * QUEUE + 2 * lane);
  int left_c = S * Rp / CH;  // chunks of the stream still to copy
  unsigned cq = 0;           // queue offset of the chunk's first entry, in bytes
  auto copy = [&]() {
    if (left_c > 0) {
#pragma unroll
      for (int u = 0; u < CH / 2; u++) {
        fetch16(queue_a + cq + u * 512, sB + u * 64);
        fetch16(queue_a + cq + QW + u * 512, sW + u * 64);
      }
      sB += CH * 32;
      sW += CH * 32;
      left_c--;
    }
    fetch_commit();
    cq = cq + CH * QE == DEPTH * QE ? 0 : cq + CH * QE;
  };
  // march coupling of this lane's position in a strip
  auto coupling = [&](int st) {
    const int c = col(st), m = FWD ? min(c, M) : max(c, 1), d = FWD ? m - 1 : m;
    return COMP == 0 ? ro(g.r2 + m) * ro(g.r2s + d) : ro(g.r1 + m) * ro(g.r1s + d);
  };

  // ---- the chain: lane t on row T - t. Before its first row, on idle steps and after its last
  // strip a lane computes what nothing reads
  float gp = 0.f, gpn = 0.f, gpl = coupling(0);  // of this lane's strip, of the one it goes over to, and the one after
  int sf = 0;  // lane 0's strip
  C v = z;
  unsigned qo = lane == 0 ? 0 : (unsigned)(DEPTH - lane) * QE;  // its queue entry
  int cf = 0;                                                    // lane 0's row at the chunk's start
  const float* const gl = rowgn + 32 - lane;
  // starting: lanes go over to the next strip in this chunk; first: from none
  auto chain = [&](auto starting, bool first) {
    C B[CH], w[CH], le[CH];
    float gn[CH];
    unsigned q[CH];
#pragma unroll
    for (int u = 0; u < CH; u++) {
      q[u] = qo;
      qo = min(qo + QE, qo - (DEPTH - 1) * QE);  // (unsigned: the second is the smaller at the queue's end)
      B[u] = *(const C*)(queue + q[u]);
      w[u] = *(const C*)(queue + q[u] + QW);
      gn[u] = gl[cf + u];
      le[u] = z;
      if (lane == 0) le[u] = edge[cf + u + 31];  // the strip before, at lane 0's row
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      C left = make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
      if constexpr (starting.value) {
        const bool now = cf + u == lane;
        gp = now ? gpn : gp;
        v.x = now ? 0.f : v.x;
        v.y = now ? 0.f : v.y;
        // lane 0 gets its own value, which gs clears, unless it comes from rows past the last,
        // whose entries hold anything
        left.x = lane == 0 ? 0.f : left.x;
        left.y = lane == 0 ? 0.f : left.y;
      }
      const float gs = lane == 0 ? 0.f : gp;
      const C d = make_float2(gp * le[u].x + gn[u] * v.x, gp * le[u].y + gn[u] * v.y);
      const C t = make_float2(d.x + gs * left.x, d.y + gs * left.y);
      v = make_float2(B[u].x + w[u].x * t.x - w[u].y * t.y, B[u].y + w[u].x * t.y + w[u].y * t.x);
      B[u] = v;
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      *(C*)(queue + q[u]) = B[u];
      if (starting.value && cf + u < 31) {  // the last rows of the strip before
        if (lane == 31 && !first) edge[cf + u + Rp] = B[u];
      } else if (lane == 31) {
        edge[cf + u] = B[u];
      }
    }
  };

  // ---- stores of the rows that the chunk has completed: 32 behind lane 0. Ex's and Ey's rows
  // are planes, the upper ones (from k0 on) in y, the lower in the cap
  const int k0 = COMP == 2 ? 0 : s.vshift;
  const long so = COMP == 0 ? (long)n1 * (n2 + 1) : (COMP == 1 ? (long)L1 * n2 : L1);
  C* const oU = COMP == 2 ? V.row(2, line, 0) : V.row(COMP, k0, COMP == 1 ? line : 0) - k0 * so;
  C* const oL = COMP == 2 || !V.CAP[COMP] ? oU : V.CAP[COMP] + (COMP == 1 ? (long)line * L1 : 0);
  int sw = 0, rw = -32;  // strip and first row
  unsigned wq = (DEPTH - 32) * QE;  // their first entry
  auto store = [&]() {
    if (rw >= 0 && rw < R) {
      if constexpr (COMP != 0) {
        const int m = col(sw);
        C o[CH];
#pragma unroll
        for (int u = 0; u < CH; u++) o[u] = *(const C*)(queue + wq + u * QE);
        if (m >= 1 && m <= M) {
#pragma unroll
          for (int u = 0; u < CH; u++) {
            const int r = row_of(rw + u);
            if (rw + u < R) ((r >= k0 ? oU : oL) + r * so)[m] = o[u];
          }
        }
      } else {
        // 32 / LINES positions of all lines for each warp
        const int t = (32 * warp + lane) / LINES, l = lane % LINES, pos = 32 * sw + t, i = line0 + l;
        if (pos < M && i < n1) {
          const long o = (long)(FWD ? 1 + pos : M - pos) * n1 + i;
          const char* const in = (const char*)(smem + l * QUEUE + t) + wq;
#pragma unroll
          for (int u = 0; u < CH; u++) {
            const int r = row_of(rw + u);
            if (rw + u < R) ((r >= k0 ? oU : oL) + r * so)[o] = *(const C*)(in + u * QE);
          }
        }
      }
    }
    rw += CH;
    if (rw == Rp) {
      rw = 0;
      sw++;
    }
    wq = wq + CH * QE == DEPTH * QE ? 0 : wq + CH * QE;
  };

  // Chunk c: the line's warp goes through it, while the other stores the rows that chunk c - 1
  // completed, copies chunk c + AHEAD into their entries and waits for chunk c + 1's.
  const int chunks = ((S - 1) * Rp + R + 32 + CH - 1) / CH;
  if (mover) {
#pragma unroll
    for (int q = 0; q < AHEAD; q++) copy();
    fetch_wait<AHEAD - 1>();
    __syncthreads();
    for (int c = 0; c < chunks; c++) {
      if (c > 0) store();
      if (LINES > 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * LINES) : "memory");
      else __syncwarp();
      copy();
      fetch_wait<AHEAD - 1>();
      __syncthreads();
    }
    store();
    fetch_wait<0>();
  } else {
    __syncthreads();
    for (int c = 0; c < chunks; c++) {
      if (cf == 0) {
        gpn = gpl;
        gpl = coupling(++sf);
      }
      if (cf < 32) chain(std::true_type(), c * CH < 32);
      else chain(std::false_type(), false);
      cf = cf + CH == Rp ? 0 : cf + CH;
      __syncthreads();
    }
  }
}

namespace {

template <int COMP, bool FWD, int NS>
void launch_pass(const SweepP<F32>& s, int sets, float2* SB, float2* SW, long sbs, const int* groups, cudaStream_t st)
{
  const int n1 = s.g.n1, n2 = s.g.n2, nK = s.nK;
  if constexpr (COMP == 0) {
    const int nti = (n1 + 32 - 1) / 32;
    dim3 grd((unsigned)(nti * sets), (unsigned)(2 * line_strips(n2 - 1)), (unsigned)(nK - 1));
    keep_l1<k_line_pass_ex<FWD, NS>>(PASS_SMEM);
    count_launch(), k_line_pass_ex<FWD, NS><<<grd, 256, 0, st>>>(s, SB, SW, sbs, nti, groups);
  } else {
    const int js = COMP == 1 ? n2 : n2 - 1, ks = COMP == 1 ? nK - 1 : nK;
    dim3 grd((unsigned)(line_strips(n1 - 1) * sets), (unsigned)((js + 2 * PASS_WARPS - 1) / (2 * PASS_WARPS)), (unsigned)ks);
    keep_l1<k_line_pass<COMP, FWD, NS>>(PASS_SMEM);
    count_launch(), k_line_pass<COMP, FWD, NS><<<grd, 32 * PASS_WARPS, 0, st>>>(s, SB, SW, sbs, groups);
  }
}
template <int COMP, bool FWD>
void launch_passes(const SweepP<F32>& s, int nslot, float2* SB, float2* SW, long sbs, const int* groups, int ngroups,
                   cudaStream_t st)
{
  if (groups) launch_pass<COMP, FWD, SPLIT_GROUP>(s, ngroups, SB, SW, sbs, groups, st);
  else launch_pass<COMP, FWD, 1>(s, nslot, SB, SW, sbs, nullptr, st);
}

template <int COMP, bool FWD, int LINES, int CH>
void launch_line_of(const SweepP<F32>& s, int nslot, const float2* SB, const float2* SW, long sbs, const int* group_of,
                    cudaStream_t st)
{
  const int R = COMP == 2 ? s.g.n2 - 1 : s.nK - 1, nlines = COMP == 0 ? s.g.n1 : (COMP == 1 ? s.g.n2 : s.nK);
  const int gps = (nlines + LINES - 1) / LINES;
  const size_t sm = line_smem<LINES, CH>(R);
  const auto kernel = k_line32<COMP, FWD, LINES, CH>;
  allow_smem<k_line32<COMP, FWD, LINES, CH>>(sm);
  count_launch(), kernel<<<(unsigned)((long)gps * nslot), 64 * LINES, sm, st>>>(s, SB, SW, sbs, group_of, gps);
}
template <int COMP, bool FWD>
void launch_line(const SweepP<F32>& s, int nslot, const float2* SB, const float2* SW, long sbs, const int* group_of,
                 cudaStream_t st)
{
  const long sms = sm_count();
  if constexpr (COMP != 0) {
    // chunks of 4 rows cost 3% more than chunks of 8, but 8 lines fit an SM instead of 7: taken
    // where that saves one of few rounds of the SMs (an application, 200 x 140 x 140 cells: 8
    // systems 2.71 -> 2.55 ms, 16 4.81 -> 4.70, 24 7.09 -> 7.00, 32 9.37 -> 9.34; 48, from 7
    // rounds to 6, 13.88 -> 13.97)
    const long lines = (long)(COMP == 1 ? s.g.n2 : s.nK) * nslot;
    const long rounds7 = (lines + 7 * sms - 1) / (7 * sms), rounds8 = (lines + 8 * sms - 1) / (8 * sms);
    if (rounds8 < rounds7 && rounds7 <= 5) launch_line_of<COMP, FWD, 1, 4>(s, nslot, SB, SW, sbs, group_of, st);
    else launch_line_of<COMP, FWD, 1, 8>(s, nslot, SB, SW, sbs, group_of, st);
  } else {
    // 8 lines to a CTA fill an SM and store 64 bytes at a time, but share its load and store unit:
    // 4 where every CTA of 4 has an SM of its own (an application, 200 x 140 x 140 cells, 8
    // against 4 lines: 2 systems 1.05 and 0.97 ms, 3 1.24 and 1.18, 4 (200 CTAs) 1.44 and 1.49)
    if ((long)((s.g.n1 + 3) / 4) * nslot <= sms) launch_line_of<0, FWD, 4, 8>(s, nslot, SB, SW, sbs, group_of, st);
    else launch_line_of<0, FWD, 8, 4>(s, nslot, SB, SW, sbs, group_of, st);
  }
}

}  // namespace

// the rows' tables, the edge columns and the queues fit shared memory, and a system's vector
// the pass's 32-bit byte offsets
bool sweep_line_fits(int n1, int n2, int nK)
{
  const double most = 8.0 * 3.0 * (n1 + 1.0) * (n2 + 1.0) * (nK + 1.0);
  return most < 4294967296.0 && n1 >= 2 && n2 >= 2 && nK >= 2 && line_smem<8, 4>(nK - 1) <= SMEM_MOST && line_smem<1, 8>(n2 - 1) <= SMEM_MOST;
}

// entries per slot: the largest component's lines as streams
long sweep_line_scratch(int n1, int n2, int nK)
{
  const int sk = line_steps(nK - 1), sj = line_steps(n2 - 1);
  const size_t a = line_entry(line_strips(n2 - 1), sk, n1, 0, 0), b = line_entry(line_strips(n1 - 1), sk, n2, 0, 0),
               c = line_entry(line_strips(n1 - 1), sj, nK, 0, 0);
  return (long)std::max(a, std::max(b, c));
}

void launch_line_bounds(const SweepP<F32>& s, int nslot, cudaStream_t st)
{
  count_launch(), k_line_bounds<<<dim3(s.nK + 1, 3, nslot), 128, 0, st>>>(s);
}

void launch_aphi_rhs(const SweepP<F32>& s, float2* T, int nslot, cudaStream_t st)
{
  count_launch(), k_aphi_rhs<<<dim3((unsigned)((s.g.lE + 255) / 256), nslot), 256, 0, st>>>(s, T);
}

void launch_line_pass(const SweepP<F32>& s, int comp, bool fwd, int nslot, float2* SB, float2* SW, long sbs,
                      const int* groups, int ngroups, cudaStream_t st)
{
  if (comp == 0) {
    if (fwd) launch_passes<0, true>(s, nslot, SB, SW, sbs, groups, ngroups, st);
    else launch_passes<0, false>(s, nslot, SB, SW, sbs, groups, ngroups, st);
  } else if (comp == 1) {
    if (fwd) launch_passes<1, true>(s, nslot, SB, SW, sbs, groups, ngroups, st);
    else launch_passes<1, false>(s, nslot, SB, SW, sbs, groups, ngroups, st);
  } else {
    if (fwd) launch_passes<2, true>(s, nslot, SB, SW, sbs, groups, ngroups, st);
    else launch_passes<2, false>(s, nslot, SB, SW, sbs, groups, ngroups, st);
  }
}

void launch_sweep_line(const SweepP<F32>& s, int comp, bool fwd, int nslot, const float2* SB, const float2* SW, long sbs,
                       const int* group_of, cudaStream_t st)
{
  if (comp == 0) {
    if (fwd) launch_line<0, true>(s, nslot, SB, SW, sbs, group_of, st);
    else launch_line<0, false>(s, nslot, SB, SW, sbs, group_of, st);
  } else if (comp == 1) {
    if (fwd) launch_line<1, true>(s, nslot, SB, SW, sbs, group_of, st);
    else launch_line<1, false>(s, nslot, SB, SW, sbs, group_of, st);
  } else {
    if (fwd) launch_line<2, true>(s, nslot, SB, SW, sbs, group_of, st);
    else launch_line<2, false>(s, nslot, SB, SW, sbs, group_of, st);
  }
}

}  // namespace csem
