// complex64 LU-SGS component sweeps as a pass over all points and a chain with a warp per
// line and no barrier.
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
// i, the axis its operands are contiguous on, so 32 x 32 tiles turn in shared memory.
//
// The chain: a warp owns one line and works through its march in strips of 32 positions, lane t on
// position t of the strip, over all rows of the strip before the next strip. Lane t runs t
// rows behind lane 0, so that lane t - 1's value at its row is there, one shuffle away, when
// it is due. Loads and stores stay together all the same: rows are copied into a queue in
// shared memory (cp.async, 16 to 23 rows early), where lane t takes its entry t steps after
// lane 0 and leaves v in its place; 31 steps after lane 0 the row is complete and is stored by
// all lanes at once. A strip's last column is kept for the left neighbours
// of the next strip's first (edge), and the strips follow one another without draining:
// lanes go over to the next strip one by one. Everything that does not happen at every row
// (the strip's start, the copies and the stores) happens every 8 rows, and the 8 rows' queue
// entries are in registers before the chain goes through them, so that a step is little more
// than the dependence: a shuffle and four multiply-adds.
//
// Ex is the contiguous axis across its lines: 8 warps take 8 neighbouring lines and store
// their rows together, 64 bytes at a time, after a barrier every 8 rows.
//
// The thread-per-row pipelines (k_sweep_ex32s, k_sweep_eyz32s, lusgs_split 1) read one 16-byte
// entry per row and lane, 20 sectors a request, and join a line's warps by barriers at every
// step. Per application, them against this, one context: 200 x 140 x 140 cells, 48 systems
// 23.3 -> 14.6 ms, 16 systems 8.02 -> 5.30, 3 systems 2.11 -> 1.40; 84^3 cells, 6 systems
// 0.86 -> 0.51; 81 x 73 x 67 cells, 3 systems at 3 frequencies 0.51 -> 0.35. The pass takes
// 60% of it, at 55% of the DRAM rate; the chain runs at 40%, bound by its steps' latency and
// the warps that shared memory leaves room for (7 on an SM).
#include <type_traits>
#include "csem_cuda.cuh"
#include "engine.h"
#include "k_sweep_common.cuh"

namespace csem {

using namespace sweep;

namespace {

typedef float2 C;

__device__ __forceinline__ C shfl(C v, int from)
{
  return make_float2(__shfl_sync(0xffffffffu, v.x, from), __shfl_sync(0xffffffffu, v.y, from));
}
__device__ __forceinline__ void fetch16(unsigned dst, const void* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int CH = 8;  // rows per chunk
// Ey, Ez: one warp to a CTA, two chunks copied ahead; Ex: 8 warps, whose shared memory leaves
// room for one
template <int COMP> struct LineShape {
  static constexpr int WARPS = COMP == 0 ? 8 : 1;
  static constexpr int AHEAD = COMP == 0 ? 1 : 2;
  static constexpr int DEPTH = 32 + CH * (1 + AHEAD);  // queue entries per lane: 32 rows in work or to be stored, and the copies
  // a warp's queue in float2: B (and then v) [DEPTH][32], w [DEPTH][32], 4 of padding (Ex's
  // lines on different banks)
  static constexpr int QUEUE = 2 * DEPTH * 32 + 4;
};
constexpr unsigned QE = 256;  // bytes from a lane's queue entry to its next

// shared memory: queues, edge columns float2 [warps][Rp + 32], row couplings float [32 + Rp]
// (the first 32: the last rows of the strip before)
template <int COMP> inline size_t line_smem(int R)
{
  const size_t Rp = line_steps(R);
  return LineShape<COMP>::WARPS * (LineShape<COMP>::QUEUE * 8 + (Rp + 32) * 8) + (Rp + 32) * 4;
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

constexpr int PASS_WARPS = 4;

}  // namespace

// Ey and Ez: a warp per strip of a row, PASS_WARPS neighbouring j. grid (strips x groups, j, k)
template <int COMP, bool FWD, int NS>
__global__ void __launch_bounds__(32 * PASS_WARPS)
    k_line_pass(SweepP<F32> s, float2* SB, float2* SW, long sbs, const int* groups)
{
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK, L1 = n1 + 1;
  const int M = n1 - 1, R = COMP == 1 ? nK - 1 : n2 - 1, S = line_strips(M), Rp = line_steps(R);
  const int grp = blockIdx.x / S, strip = blockIdx.x - grp * S;
  const int lane = threadIdx.x & 31, j = blockIdx.y * PASS_WARPS + (threadIdx.x >> 5) + (COMP == 2 ? 1 : 0);
  const int k = blockIdx.z + (COMP == 1 ? 1 : 0);
  const int p = strip * 32 + lane, i = FWD ? min(1 + p, M) : max(M - p, 1);
  const Members<NS> mem(s, groups, grp);
  const SysScal<F32> sc = s.scal[mem.sys_of(0)];
  if (j >= n2) return;
  const bool on = p < M;  // (lanes past the last position form position M again, and store nothing)
  // Ey: row axis Z (k), line axis Y (j); Ez: row axis Y (j), line axis Z (k)
  const Ax<F32> Rw = COMP == 1 ? axis<F32>(g.d3, g.d3s, g.r3, g.r3s, k) : axis<F32>(g.d2, g.d2s, g.r2, g.r2s, j);
  const Ax<F32> LA = COMP == 1 ? axis_at<F32>(g.d2, g.d2s, g.r2, g.r2s, j) : axis_at<F32>(g.d3, g.d3s, g.r3, g.r3s, k);
  const Ax<F32> X = axis<F32>(g.d1, g.d1s, g.r1, g.r1s, i);
  const float gg = (X.rs + X.rsm) * X.r + (Rw.rs + Rw.rsm) * Rw.r;  // geo(Z, X) / geo(X, Y)
  const float ydd = COMP == 1 ? LA.d : Rw.d, zdd = COMP == 1 ? Rw.d : LA.d;
  const float sg = ro(COMP == 1 ? g.s22 + ix2(n1, n2, k, j, i) : g.s33 + ix3(n1, n2, k, j, i));
  const Coef32 cf = lin_coef(sc, g.fvm, gg, sg, X.ds * ydd * zdd);
  const size_t e = line_entry(S, Rp, COMP == 1 ? j : k, p, COMP == 1 ? (FWD ? k - 1 : R - k) : (FWD ? j - 1 : R - j));
  if (on) SW[(size_t)grp * sbs + e] = cf.w;
  const int kB = COMP == 1 ? k - 1 : k + 1;
  const bool upA = k >= s.vshift, upB = kB >= s.vshift;
  // Ex and the third component either side of the line, own old values on the lower side
  const unsigned xb = 8u * (unsigned)(plane(s, 0, k, upA) + (long)j * n1 + i);
  const unsigned xa = COMP == 1 ? xb + 8u * n1 : 8u * (unsigned)(plane(s, 0, kB, upB) + (long)j * n1 + i);
  unsigned ya, yb, yc, yd;  // upper and lower side of the line, at the row and at the row below
  if (COMP == 1) {
    yb = 8u * (unsigned)(plane(s, 2, k, upA) + (long)j * L1 + i), ya = yb + 8u * L1;
    yd = 8u * (unsigned)(plane(s, 2, kB, upB) + (long)j * L1 + i), yc = yd + 8u * L1;
  } else {
    yb = 8u * (unsigned)(plane(s, 1, k, upA) + (long)j * L1 + i), yd = yb - 8u * L1;
    ya = 8u * (unsigned)(plane(s, 1, kB, upB) + (long)j * L1 + i), yc = ya - 8u * L1;
  }
  const unsigned own = 8u * (unsigned)(plane(s, COMP, k, upA) + (long)j * L1 + i);
  const unsigned low = COMP == 1 ? 8u * (unsigned)(plane(s, 1, kB, upB) + (long)j * L1 + i) : own - 8u * L1;
  const float km = X.r * X.rsm, kr = Rw.r * Rw.rsm;
  const C z = make_float2(0.f, 0.f);
  float2* out = SB + e;
  struct Vals {
    C b, xa, xb, xc, xd, ya, yb, yc, yd, o, lo;
  };
  auto load = [&](int q) {
    const Bases m = bases(s, mem.slot_of(q), mem.sys_of(q), upA, upB);
    const char* const xA = COMP == 1 ? m.A : m.B;
    Vals v;
    v.b = upA ? at(m.x, own) : z;
    v.xa = at(xA, xa), v.xb = at(m.A, xb), v.xc = at(xA, xa - 8), v.xd = at(m.A, xb - 8);
    if (COMP == 2 || !FWD) {
      v.ya = at(COMP == 1 ? m.A : m.B, ya), v.yb = at(m.A, yb);
      v.yc = at(m.B, yc), v.yd = at(COMP == 1 ? m.B : m.A, yd);
    }
    if (!FWD) v.o = at(m.A, own - 8), v.lo = at(COMP == 1 ? m.B : m.A, low);
    return v;
  };
  auto form = [&](int q, const Vals& v) {
    const C dx = sub32(sub32(v.xa, v.xb), sub32(v.xc, v.xd));
    // Ey: Y.rs (Z.r dEz + X.r dEx); Ez: Z.rs (X.r dEx + Y.r dEy)
    C acc = scl32(X.r, dx);
    if (COMP == 2 || !FWD) {
      const C dy = sub32(sub32(v.ya, v.yb), sub32(v.yc, v.yd));
      acc = make_float2(acc.x + Rw.r * dy.x, acc.y + Rw.r * dy.y);
    }
    C kc = scl32(-LA.rs, acc);
    if (!FWD) kc = make_float2(kc.x + (km * v.o.x + kr * v.lo.x), kc.y + (km * v.o.y + kr * v.lo.y));
    const C B = lin_B(cf, g.fvm, v.b, kc);
    const int slot = mem.slot_of(q);
    if (on) out[(size_t)slot * sbs] = B;
  };
  int q = 0;
  for (; q + 1 < mem.n; q += 2) {  // two systems' loads in flight
    const Vals v = load(q), u = load(q + 1);
    form(q, v);
    form(q + 1, u);
  }
  if (q < mem.n) form(q, load(q));
}

// Ex: a CTA forms 32 i x a strip's 32 positions j, along i, and stores them along j.
// grid (i tiles x groups, strips, k)
template <bool FWD, int NS>
__global__ void __launch_bounds__(512) k_line_pass_ex(SweepP<F32> s, float2* SB, float2* SW, long sbs, int nti, const int* groups)
{
  __shared__ C tiles[2][32][33];  // one is written while the other's values go out
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
  Coef32 cf[2];
  float yr[2], kj[2];
  unsigned ox[2], oy[2], oz[2], ozm[2], oxm[2];
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const int st = 32 * blockIdx.y + ty + 16 * a, j = FWD ? min(1 + st, M) : max(M - st, 1);  // (past the last position: it again)
    const Ax<F32> Y = axis<F32>(g.d2, g.d2s, g.r2, g.r2s, j);
    const float gg = (Y.rs + Y.rsm) * Y.r + (Z.rs + Z.rsm) * Z.r;  // geo(Y, Z)
    cf[a] = lin_coef(sc, g.fvm, gg, ro(g.s11 + ix1(n1, n2, k, j, i)), xds * Y.d * Z.d);
    yr[a] = Y.r;
    kj[a] = Y.r * Y.rsm;
    ox[a] = 8u * (unsigned)(plane(s, 0, k, upA) + (long)j * n1 + i);
    oxm[a] = 8u * (unsigned)(plane(s, 0, k - 1, upB) + (long)j * n1 + i);
    oy[a] = 8u * (unsigned)(plane(s, 1, k, upA) + (long)j * L1 + i);
    oz[a] = 8u * (unsigned)(plane(s, 2, k, upA) + (long)j * L1 + i);
    ozm[a] = 8u * (unsigned)(plane(s, 2, k - 1, upB) + (long)j * L1 + i);
    tiles[1][ty + 16 * a][tx] = cf[a].w;
  }
  const size_t e0 = line_entry(S, Rp, i0 + ty, 32 * blockIdx.y + tx, FWD ? k - 1 : R - k), e1 = line_entry(S, Rp, 16, 0, 0);
  const bool w0 = i0 + ty < n1, w1 = i0 + ty + 16 < n1;
  auto turn = [&](C(*tile)[33], C* out) {
    __syncthreads();
    if (w0) out[e0] = tile[tx][ty];
    if (w1) out[e0 + e1] = tile[tx][ty + 16];
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
    C(*tile)[33] = tiles[q & 1];
#pragma unroll
    for (int a = 0; a < 2; a++) {
      C kc = z;
      if (!FWD) {
        const C dy = sub32(sub32(v[a].ya, v[a].yb), sub32(v[a].yc, v[a].yd));
        const C dz = sub32(sub32(v[a].za, v[a].zb), sub32(v[a].zc, v[a].zd));
        const C cross = scl32(xrs, make_float2(yr[a] * dy.x + Z.r * dz.x, yr[a] * dy.y + Z.r * dz.y));
        kc = sub32(make_float2(kj[a] * v[a].ej.x + kz * v[a].ek.x, kj[a] * v[a].ej.y + kz * v[a].ek.y), cross);
      }
      tile[ty + 16 * a][tx] = lin_B(cf[a], g.fvm, v[a].b, kc);
    }
    if (q + 1 < mem.n) load(q + 1);  // in flight while this system's tile turns
    turn(tile, SB + (size_t)mem.slot_of(q) * sbs);
  }
}

template <int COMP, bool FWD>
__global__ void __launch_bounds__(32 * LineShape<COMP>::WARPS) k_line32(SweepP<F32> s, const float2* SB, const float2* SW,
                                                                        long sbs, const int* group_of, int groups_per_slot)
{
  constexpr int WARPS = LineShape<COMP>::WARPS, AHEAD = LineShape<COMP>::AHEAD, DEPTH = LineShape<COMP>::DEPTH,
                QUEUE = LineShape<COMP>::QUEUE;
  constexpr unsigned QW = DEPTH * QE;  // bytes from a B to its w
  extern __shared__ float2 smem[];
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK;
  const int nlines = COMP == 0 ? n1 : (COMP == 1 ? n2 : nK);
  const int R = COMP == 2 ? n2 - 1 : nK - 1;  // rows 1..R
  const int M = COMP == 0 ? n2 - 1 : n1 - 1;  // march positions 1..M
  const int Rp = line_steps(R);
  const int S = (M + 31) / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = blockIdx.x / groups_per_slot;
  const int line0 = (blockIdx.x - slot * groups_per_slot) * WARPS;
  const int line = WARPS > 1 ? min(line0 + warp, nlines - 1) : line0;  // (a CTA's warps stay together)
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  const View<F32> V = view_of<F32>(s, slot, sys);
  const C z = make_float2(0.f, 0.f);
  const int L1 = n1 + 1;
  auto row_of = [&](int rho) { return FWD ? 1 + rho : R - rho; };
  auto col = [&](int st) { return FWD ? 1 + 32 * st + lane : M - 32 * st - lane; };

  C* const edge = smem + WARPS * QUEUE + warp * (Rp + 32);
  float* const rowgn = (float*)(smem + WARPS * QUEUE + WARPS * (Rp + 32));
  // what couples a step's row to the row before
  for (int q = threadIdx.x; q < 32 + Rp; q += 32 * WARPS) {
    const int rho = q < 32 ? q - 32 + Rp : q - 32;
    float gn = 0.f;
    if (rho < R) {
      const int r = row_of(rho), d = FWD ? r - 1 : r;
      gn = COMP == 2 ? ro(g.r2 + r) * ro(g.r2s + d) : ro(g.r3 + r) * ro(g.r3s + d);
    }
    rowgn[q] = gn;
  }
  for (int q = lane; q < Rp + 32; q += 32) edge[q] = z;
  __syncthreads();

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
      le[u] = edge[cf + u + 31];  // the strip before, at lane 0's row
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      C left = shfl(v, lane - 1);
      left.x = lane == 0 ? le[u].x : left.x;
      left.y = lane == 0 ? le[u].y : left.y;
      if constexpr (starting.value) {
        const bool now = cf + u == lane;
        gp = now ? gpn : gp;
        v.x = now ? 0.f : v.x;
        v.y = now ? 0.f : v.y;
      }
      const C t = make_float2(gp * left.x + gn[u] * v.x, gp * left.y + gn[u] * v.y);
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
  int sw = 0, rw = -32;
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
        // this warp's row of the chunk: 4 positions of 8 lines at a time
        const int i = line0 + (lane & 7), r = row_of(rw + warp);
        if (rw + warp < R && i < n1) {
          C* const out = (r >= k0 ? oU : oL) + r * so + i;
          const char* const in = (const char*)(smem + (lane & 7) * QUEUE) + wq + warp * QE;
#pragma unroll
          for (int a = 0; a < 8; a++) {
            const int t = a * 4 + (lane >> 3), m = FWD ? 1 + 32 * sw + t : M - 32 * sw - t;
            if (m >= 1 && m <= M) out[(long)m * n1] = *(const C*)(in + t * 8);
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

#pragma unroll
  for (int q = 0; q < AHEAD; q++) copy();
  const int chunks = ((S - 1) * Rp + R + 32 + CH - 1) / CH;
  for (int c = 0; c < chunks; c++) {
    if (cf == 0) {
      gpn = gpl;
      gpl = coupling(++sf);
    }
    fetch_wait<AHEAD - 1>();
    __syncwarp();  // the other lanes' copies are there, too
    copy();
    if (cf < 32) chain(std::true_type(), c < 4);
    else chain(std::false_type(), false);
    cf = cf + CH == Rp ? 0 : cf + CH;
    if (WARPS > 1) __syncthreads();  // every line has its part of the rows
    else __syncwarp();               // edge
    store();
    if (WARPS > 1) __syncthreads();  // before the next copies take the entries
  }
  fetch_wait<0>();
}

namespace {

template <int COMP, bool FWD, int NS>
void launch_pass(const SweepP<F32>& s, int sets, float2* SB, float2* SW, long sbs, const int* groups, cudaStream_t st)
{
  const int n1 = s.g.n1, n2 = s.g.n2, nK = s.nK;
  if constexpr (COMP == 0) {
    const int nti = (n1 + 31) / 32;
    dim3 grd((unsigned)(nti * sets), (unsigned)line_strips(n2 - 1), (unsigned)(nK - 1));
    count_launch(), k_line_pass_ex<FWD, NS><<<grd, 512, 0, st>>>(s, SB, SW, sbs, nti, groups);
  } else {
    const int js = COMP == 1 ? n2 : n2 - 1, ks = COMP == 1 ? nK - 1 : nK;
    dim3 grd((unsigned)(line_strips(n1 - 1) * sets), (unsigned)((js + PASS_WARPS - 1) / PASS_WARPS), (unsigned)ks);
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

template <int COMP, bool FWD>
void launch_line(const SweepP<F32>& s, int nslot, const float2* SB, const float2* SW, long sbs, const int* group_of,
                 cudaStream_t st)
{
  constexpr int W = LineShape<COMP>::WARPS;
  const int R = COMP == 2 ? s.g.n2 - 1 : s.nK - 1, nlines = COMP == 0 ? s.g.n1 : (COMP == 1 ? s.g.n2 : s.nK);
  const int gps = (nlines + W - 1) / W;
  const size_t sm = line_smem<COMP>(R);
  allow_smem<k_line32<COMP, FWD>>(sm);
  count_launch(), k_line32<COMP, FWD><<<(unsigned)((long)gps * nslot), 32 * W, sm, st>>>(s, SB, SW, sbs, group_of, gps);
}

}  // namespace

// the rows' tables, the edge columns and the queues fit shared memory, and a system's vector
// the pass's 32-bit byte offsets
bool sweep_line_fits(int n1, int n2, int nK)
{
  const double most = 8.0 * 3.0 * (n1 + 1.0) * (n2 + 1.0) * (nK + 1.0);
  return most < 4294967296.0 && n1 >= 2 && n2 >= 2 && nK >= 2 && line_smem<0>(nK - 1) <= SMEM_MOST && line_smem<1>(nK - 1) <= SMEM_MOST &&
         line_smem<2>(n2 - 1) <= SMEM_MOST;
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
