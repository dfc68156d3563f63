// complex64 LU-SGS component sweeps as lockstep row pipelines: one launch per sweep.
//
// A sweep updates one field component in the reference's lexicographic Gauss-Seidel
// order (fdfd.c:347-503). In the coupled plane (r, m) a point depends on (r-1, m) and
// (r, m-1) (forward; (r+1, m), (r, m+1) backward); the third axis is independent:
//   Ex: rows r = k, march m = j, independent i  (VW consecutive i per lane)
//   Ey: rows r = k, march m = i, independent j  (VW consecutive i per step)
//   Ez: rows r = j, march m = i, independent k  (VW consecutive i per step)
// One CTA owns one independent line of one system and gives every row of the sweep a
// thread: thread t takes the t-th row in sweep order. All rows advance together, one
// march step per iteration, skewed by one step per row: at step T row t works at march
// position T - t, so the row before it finished that position at step T - 1. That value
// arrives by warp shuffle, or through shared memory from the last lane of the previous
// warp (pairwise named barriers between neighbouring warps). The own-row dependency stays
// in registers and the sweep's first row depends on the boundary, which is zero. A sweep
// takes (march positions + rows - 1) steps.
//
// Every point is evaluated in linear form, with reciprocal spacings (below); k_lusgs64.cu
// has the complex128 sweeps, which keep the reference's operations.
#include "csem_cuda.cuh"
#include "engine.h"
#include "k_sweep_common.cuh"

namespace csem {

using namespace sweep;

namespace {

// resident CTAs per SM the register budget is sized for, by points per thread and step
template <int VW> struct MinBlocks {
  static constexpr int value = VW >= 4 ? 1 : (VW == 2 ? 2 : 3);
};
// Register budget of the sweeps: by default from MinBlocks for a full CTA; a build may set
// explicit caps per width (CSEM_SWEEP_MAXNREG1 / 2 / 4) for CTAs of up to 256 rows instead.
#if defined(CSEM_SWEEP_MAXNREG1) && defined(CSEM_SWEEP_MAXNREG2) && defined(CSEM_SWEEP_MAXNREG4)
template <int VW> struct RegCap {
  static constexpr int value = VW == 1 ? CSEM_SWEEP_MAXNREG1 : (VW == 2 ? CSEM_SWEEP_MAXNREG2 : CSEM_SWEEP_MAXNREG4);
};
#define CSEM_SWEEP_BOUNDS32(VW, MAXR) __launch_bounds__(MAXR) __maxnreg__(MAXR > NB_ROWS ? 128 : RegCap<VW>::value)
#else
#define CSEM_SWEEP_BOUNDS32(VW, MAXR) __launch_bounds__(MAXR, MAXR > NB_ROWS ? 1 : MinBlocks<VW>::value)
#endif

}  // namespace

// ---------------------------------------------------------------------------------------
// complex64 sweeps: linear form, operands one step ahead.
//
// The update of a point is linear in the values it takes from the chain: its own row at
// the previous march position (prev) and the previous row at this position (nb). With
// the component's own point zero while its row is evaluated (fdfd.c:357,383,409), the
// reference's update (b - aij) / aii rearranges to
//   v = B + w (gp prev + gn nb),  w = iwmu / aii,
//   B = b / (f aii) + w (known - cross),
// where cross is the coupling to the other two components (read-only during the sweep),
// known the own-component neighbours already fixed when the point is reached (the
// not-yet-swept values of the backward sweep), gp and gn the spacing products of the two
// chain neighbours and f = vol iom with fvm (1 otherwise). B, w, gp, gn depend only on
// operands no other thread of the sweep writes before the point is reached, so each step
// loads the next step's operands first, runs the short chain part (a real and a complex
// multiply-add after nb arrives), hands over, and only then folds the loaded operands
// into the next step's B and w while the loads were in flight. Same operations as the
// reference up to the order of rounding.
namespace {

// operands of one Ex step (the backward-only ones are dropped by the compiler forward)
template <int VW> struct RawEx {
  float2 b[VW], exjm[VW], exkm[VW], eyA[VW], eyB[VW], eyC[VW], eyD[VW], ezA[VW], ezB[VW], ezC[VW], ezD[VW];
  float sg[VW];
  Ax<F32> Y;
};

template <int VW> struct RawEyz {
  float2 b[VW], xA[VW], xB[VW], xC[VW], xD[VW], yA[VW], yB[VW], yC[VW], yD[VW], own2[VW], rowold[VW];
  float sg[VW];
  Ax<F32> X[VW];
};

}  // namespace

// Ex, complex64: rows k, march j, VW consecutive i per thread. grid (line groups, systems).
//
// A CTA may carry several lines one after the other (lpc lines, a conveyor): a row that
// finishes its march on one line starts the next line at the next step, while the rows
// behind it are still on the previous one. Row t works at step T on conveyor position
// u = T - t, i.e. line u / M, march position u % M, so the row before it finished the
// same line and position at step T - 1 and the hand-over is unchanged. The pipeline
// fills and drains once per CTA instead of once per line.
template <bool FWD, int VW, int MAXR>
__global__ void CSEM_SWEEP_BOUNDS32(VW, MAXR) k_sweep_ex32(SweepP<F32> s, int lpc)
{
  typedef float2 C;
  __shared__ HandOff<VW, C, (MAXR <= NB_ROWS)> hand;
  const int slot = blockIdx.y;
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK;
  const int nlines = (n1 + VW - 1) / VW;
  const int line0 = blockIdx.x * lpc;
  const int nl = min(lpc, nlines - line0);
  const View<F32> V = view_of<F32>(s, slot, sys);
  const SysScal<F32> sc = s.scal[sys];
  const C z = make_float2(0.f, 0.f);
  const int R_ = nK - 1, M = n2 - 1;  // rows k = 1..R_, march j = 1..M
  const int U = nl * M;               // conveyor positions
  const int rr = threadIdx.x;
  const bool rowok = rr < R_;
  const int k = FWD ? 1 + rr : R_ - rr;
  const Ax<F32> Z = rowok ? axis<F32>(g.d3, g.d3s, g.r3, g.r3s, k) : Ax<F32>{};
  // the row's planes at i = 0; a line adds its first i
  C* ex0 = nullptr;
  const C *ex1 = nullptr, *ey0 = nullptr, *ez0 = nullptr, *ez1 = nullptr, *bb = nullptr;
  const float* sg0 = nullptr;
  if (rowok) {
    ex0 = V.row(0, k, 0);
    ex1 = V.row(0, k - 1, 0);
    ey0 = V.row(1, k, 0);
    ez0 = V.row(2, k, 0);
    ez1 = V.row(2, k - 1, 0);
    bb = V.brow(0, k, 0);
    sg0 = g.s11 + ix1(n1, n2, k, 0, 0);
  }
  const int L1 = n1 + 1;
  const float gn = Z.r * (FWD ? Z.rsm : Z.rs);
  int il = line0 * VW;  // first i of the line the loads are on
  int is = il;          // first i of the line the stores are on
  Ax<F32> X[VW];        // spacings of the load line's i's
  auto set_line = [&](int i0) {
    il = i0;
#pragma unroll
    for (int q = 0; q < VW; q++) X[q] = i0 + q < n1 ? axis_at<F32>(g.d1, g.d1s, g.r1, g.r1s, i0 + q) : Ax<F32>{};
  };
  set_line(il);
  RawEx<VW> raw;
  Lin32 lin[VW];
  // loads of march position c of the load line (nothing read here is written before that step)
  auto load = [&](int c) {
    const int j = FWD ? 1 + c : M - c;
    raw.Y = axis<F32>(g.d2, g.d2s, g.r2, g.r2s, j);
    const int ox = j * n1 + il, oy = j * L1 + il;
#pragma unroll
    for (int q = 0; q < VW; q++) {
      if (il + q < n1) {
        raw.b[q] = bb ? ro(bb + ox + q) : z;
        raw.sg[q] = ro(sg0 + ox + q);
        if (!FWD) {
          raw.exjm[q] = ex0[ox - n1 + q];
          raw.exkm[q] = ex1[ox + q];
          raw.eyA[q] = ro(ey0 + oy + q + 1);
          raw.eyB[q] = ro(ey0 + oy + q);
          raw.eyC[q] = ro(ey0 + oy - L1 + q + 1);
          raw.eyD[q] = ro(ey0 + oy - L1 + q);
          raw.ezA[q] = ro(ez0 + oy + q + 1);
          raw.ezB[q] = ro(ez0 + oy + q);
          raw.ezC[q] = ro(ez1 + oy + q + 1);
          raw.ezD[q] = ro(ez1 + oy + q);
        }
      }
    }
  };
  auto make = [&]() {
    const Ax<F32>& Y = raw.Y;
    const float gg = (Y.rs + Y.rsm) * Y.r + (Z.rs + Z.rsm) * Z.r;  // geo(Y, Z)
    const float gp = Y.r * (FWD ? Y.rsm : Y.rs);
#pragma unroll
    for (int q = 0; q < VW; q++) {
      if (il + q >= n1) continue;
      C kc = z;
      if (!FWD) {
        const C dy = sub32(sub32(raw.eyA[q], raw.eyB[q]), sub32(raw.eyC[q], raw.eyD[q]));
        const C dz = sub32(sub32(raw.ezA[q], raw.ezB[q]), sub32(raw.ezC[q], raw.ezD[q]));
        const C cross = scl32(X[q].rs, make_float2(Y.r * dy.x + Z.r * dz.x, Y.r * dy.y + Z.r * dz.y));
        const C known = make_float2(Y.r * Y.rsm * raw.exjm[q].x + Z.r * Z.rsm * raw.exkm[q].x,
                                    Y.r * Y.rsm * raw.exjm[q].y + Z.r * Z.rsm * raw.exkm[q].y);
        kc = sub32(known, cross);
      }
      lin[q] = lin_make(sc, g.fvm, gg, raw.sg[q], X[q].ds * Y.d * Z.d, raw.b[q], kc, gp, gn);
    }
  };
  C res[VW];
#pragma unroll
  for (int q = 0; q < VW; q++) res[q] = z;
  if (rowok && rr == 0 && U > 0) {
    load(0);
    make();
  }
  for (int T = 0; T < U + R_ - 1; T++) {
    const int u = T - rr;
    const bool act = rowok && u >= 0 && u < U;
    const bool nxt = rowok && u + 1 >= 0 && u + 1 < U;
    int cn = 0;
    if (nxt) {
      cn = (u + 1) % M;
      if (cn == 0 && u + 1 > 0) set_line((line0 + (u + 1) / M) * VW);  // the loads move to the next line
      load(cn);
    }
    C nb[VW];
    hand.get(res, nb, T);
    if (act) {
      const int c = u % M;
      const int ox = (FWD ? 1 + c : M - c) * n1 + is;
#pragma unroll
      for (int q = 0; q < VW; q++) {
        if (is + q >= n1) {
          res[q] = z;
          continue;
        }
        const C v = lin_apply(lin[q], c > 0 ? res[q] : z, nb[q]);  // prev: own row, previous j
        ex0[ox + q] = v;
        res[q] = v;
      }
      if (c == M - 1) is = il;  // the stores follow the loads onto the next line
    } else {
#pragma unroll
      for (int q = 0; q < VW; q++) res[q] = z;
    }
    hand.put(res, T);
    if (nxt) make();
  }
  hand.finish(U + R_ - 1);
}

// Ey (COMP 1: line j, rows k) / Ez (COMP 2: line k, rows j), complex64: march i in
// chunks of VW, lpc lines per CTA as a conveyor (see k_sweep_ex32). grid (line groups,
// systems)
template <int COMP, bool FWD, int VW, int MAXR>
__global__ void CSEM_SWEEP_BOUNDS32(VW, MAXR) k_sweep_eyz32(SweepP<F32> s, int lpc)
{
  typedef float2 C;
  __shared__ HandOff<VW, C, (MAXR <= NB_ROWS)> hand;
  const int slot = blockIdx.y;
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  const GridP<F32>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK;
  const int nlines = COMP == 1 ? n2 : nK;
  const int line0 = blockIdx.x * lpc;
  const int nl = min(lpc, nlines - line0);
  const View<F32> V = view_of<F32>(s, slot, sys);
  const SysScal<F32> sc = s.scal[sys];
  const C z = make_float2(0.f, 0.f);
  const int R_ = COMP == 1 ? nK - 1 : n2 - 1;  // rows k (Ey) or j (Ez) = 1..R_
  const int M = n1 - 1;                         // march i = 1..M
  const int NC = (M + VW - 1) / VW;
  const int U = nl * NC;  // conveyor positions
  const int rr = threadIdx.x;
  const bool rowok = rr < R_;
  const int r = FWD ? 1 + rr : R_ - rr;
  // the row's axis (Z for Ey, Y for Ez) is fixed; the line's axis (Y for Ey, Z for Ez)
  // moves with the conveyor
  const Ax<F32> Rw = rowok ? (COMP == 1 ? axis<F32>(g.d3, g.d3s, g.r3, g.r3s, r) : axis<F32>(g.d2, g.d2s, g.r2, g.r2s, r))
                           : Ax<F32>{};
  const float gn = Rw.r * (FWD ? Rw.rsm : Rw.rs);
  // the rows the loads read (element i is row[i]) and the line's spacings
  C* own = nullptr;
  const C *nxt = nullptr, *xa = nullptr, *xb = nullptr, *ya = nullptr, *yb = nullptr, *yc = nullptr, *yd = nullptr;
  const C* bb = nullptr;
  const float* sg0 = nullptr;
  float lrs = 0.f, ld = 0.f;  // the line axis' rs (the coefficient of the line-axis differences) and d
  auto set_line = [&](int line) {
    const int k = COMP == 1 ? r : line;
    const int j = COMP == 1 ? line : r;
    const Ax<F32> LA = COMP == 1 ? axis_at<F32>(g.d2, g.d2s, g.r2, g.r2s, j) : axis_at<F32>(g.d3, g.d3s, g.r3, g.r3s, k);
    lrs = LA.rs;
    ld = LA.d;
    if (COMP == 1) {
      own = V.row(1, k, j);
      nxt = V.row(1, k - 1, j);
      xa = V.row(0, k, j + 1);
      xb = V.row(0, k, j);
      ya = V.row(2, k, j + 1);
      yb = V.row(2, k, j);
      yc = V.row(2, k - 1, j + 1);
      yd = V.row(2, k - 1, j);
      sg0 = g.s22 + ix2(n1, n2, k, j, 0);
    } else {
      own = V.row(2, k, j);
      nxt = V.row(2, k, j - 1);
      xa = V.row(0, k + 1, j);
      xb = V.row(0, k, j);
      ya = V.row(1, k + 1, j);
      yb = V.row(1, k, j);
      yc = V.row(1, k + 1, j - 1);
      yd = V.row(1, k, j - 1);
      sg0 = g.s33 + ix3(n1, n2, k, j, 0);
    }
    bb = V.brow(COMP, k, j);
  };
  if (rowok) set_line(line0);
  C* own_st = own;  // the row the stores go to (the loads run one position ahead)
  RawEyz<VW> raw;
  Lin32 lin[VW];
  auto load = [&](int c) {
#pragma unroll
    for (int q = 0; q < VW; q++) {
      const int m = c * VW + q;
      if (m < M) {
        const int i = FWD ? 1 + m : M - m;
        raw.X[q] = axis<F32>(g.d1, g.d1s, g.r1, g.r1s, i);
        raw.b[q] = bb ? ro(bb + i) : z;
        raw.sg[q] = ro(sg0 + i);
        raw.xA[q] = ro(xa + i);
        raw.xB[q] = ro(xb + i);
        raw.xC[q] = ro(xa + i - 1);
        raw.xD[q] = ro(xb + i - 1);
        if (COMP == 2 || !FWD) {
          raw.yA[q] = ro(ya + i);
          raw.yB[q] = ro(yb + i);
          raw.yC[q] = ro(yc + i);
          raw.yD[q] = ro(yd + i);
        }
        if (!FWD) {
          raw.own2[q] = own[i - 1];
          raw.rowold[q] = nxt[i];
        }
      }
    }
  };
  auto make = [&](int c) {
#pragma unroll
    for (int q = 0; q < VW; q++) {
      if (c * VW + q >= M) continue;
      const Ax<F32>& X = raw.X[q];
      const float gg = (X.rs + X.rsm) * X.r + (Rw.rs + Rw.rsm) * Rw.r;  // geo(Z, X) / geo(X, Y)
      const C dx = sub32(sub32(raw.xA[q], raw.xB[q]), sub32(raw.xC[q], raw.xD[q]));
      // Ey: Y.rs (Z.r dEz + X.r dEx); Ez: Z.rs (X.r dEx + Y.r dEy)
      C acc = scl32(X.r, dx);
      if (COMP == 2 || !FWD) {
        const C dy = sub32(sub32(raw.yA[q], raw.yB[q]), sub32(raw.yC[q], raw.yD[q]));
        acc = make_float2(acc.x + Rw.r * dy.x, acc.y + Rw.r * dy.y);
      }
      C kc = scl32(-lrs, acc);
      if (!FWD) {
        const C known = make_float2(X.r * X.rsm * raw.own2[q].x + Rw.r * Rw.rsm * raw.rowold[q].x,
                                    X.r * X.rsm * raw.own2[q].y + Rw.r * Rw.rsm * raw.rowold[q].y);
        kc = make_float2(kc.x + known.x, kc.y + known.y);
      }
      const float yd = COMP == 1 ? ld : Rw.d, zd = COMP == 1 ? Rw.d : ld;  // Y.d and Z.d
      lin[q] = lin_make(sc, g.fvm, gg, raw.sg[q], X.ds * yd * zd, raw.b[q], kc, X.r * (FWD ? X.rsm : X.rs), gn);
    }
  };
  C res[VW];
#pragma unroll
  for (int q = 0; q < VW; q++) res[q] = z;
  if (rowok && rr == 0 && U > 0) {
    load(0);
    make(0);
  }
  for (int T = 0; T < U + R_ - 1; T++) {
    const int u = T - rr;
    const bool act = rowok && u >= 0 && u < U;
    const bool nx = rowok && u + 1 >= 0 && u + 1 < U;
    int cn = 0;
    if (nx) {
      cn = (u + 1) % NC;
      if (cn == 0 && u + 1 > 0) set_line(line0 + (u + 1) / NC);  // the loads move to the next line
      load(cn);
    }
    C nb[VW];
    hand.get(res, nb, T);
    if (act) {
      const int c = u % NC;
      C prev = c > 0 ? res[VW - 1] : z;  // own row at the previous march position
#pragma unroll
      for (int q = 0; q < VW; q++) {
        const int m = c * VW + q;
        if (m >= M) {
          res[q] = z;
          continue;
        }
        const C v = lin_apply(lin[q], prev, nb[q]);
        own_st[FWD ? 1 + m : M - m] = v;
        res[q] = v;
        prev = v;
      }
      if (c == NC - 1) own_st = own;  // the stores follow the loads onto the next line
    } else {
#pragma unroll
      for (int q = 0; q < VW; q++) res[q] = z;
    }
    hand.put(res, T);
    if (nx) make(cn);
  }
  hand.finish(U + R_ - 1);
}

bool sweep_pipelined_fits(int comp, int n1, int n2, int nK)
{
  const int rows = comp == 2 ? n2 - 1 : nK - 1;
  return rows >= 1 && rows <= MAXROWS && n1 >= 2 && n2 >= 2;
}

template <int VW, int MAXR>
static void launch_vw(const SweepP<F32>& s, int comp, bool fwd, int nslot, cudaStream_t st, int lpc)
{
  const int n1 = s.g.n1, n2 = s.g.n2, nK = s.nK;
  const int rows = comp == 2 ? n2 - 1 : nK - 1;
  const int threads = (rows + 31) / 32 * 32;
  if (comp == 0) {
    dim3 grd(((n1 + VW - 1) / VW + lpc - 1) / lpc, nslot);
    if (fwd) count_launch(), k_sweep_ex32<true, VW, MAXR><<<grd, threads, 0, st>>>(s, lpc);
    else count_launch(), k_sweep_ex32<false, VW, MAXR><<<grd, threads, 0, st>>>(s, lpc);
  } else if (comp == 1) {
    dim3 grd((n2 + lpc - 1) / lpc, nslot);
    if (fwd) count_launch(), k_sweep_eyz32<1, true, VW, MAXR><<<grd, threads, 0, st>>>(s, lpc);
    else count_launch(), k_sweep_eyz32<1, false, VW, MAXR><<<grd, threads, 0, st>>>(s, lpc);
  } else {
    dim3 grd((nK + lpc - 1) / lpc, nslot);
    if (fwd) count_launch(), k_sweep_eyz32<2, true, VW, MAXR><<<grd, threads, 0, st>>>(s, lpc);
    else count_launch(), k_sweep_eyz32<2, false, VW, MAXR><<<grd, threads, 0, st>>>(s, lpc);
  }
}

// vw: points per thread and step (1, 2 or 4; other values select 2, the fastest measured
// on a 200x140x140 grid). Sweeps of more than 256 rows run 1 or 2 points per thread in CTAs
// of up to 512 threads. lines_per_cta: lines one CTA carries as a conveyor (>= 1).
void launch_sweep_pipelined(const SweepP<F32>& s, int comp, bool fwd, int nslot, cudaStream_t st, int vw,
                            int lines_per_cta)
{
  if (vw != 1 && vw != 2 && vw != 4) vw = 2;
  const int lpc = lines_per_cta > 1 ? lines_per_cta : 1;
  const int rows = comp == 2 ? s.g.n2 - 1 : s.nK - 1;
  if (rows > NB_ROWS) {
    if (vw == 1) launch_vw<1, MAXROWS>(s, comp, fwd, nslot, st, lpc);
    else launch_vw<2, MAXROWS>(s, comp, fwd, nslot, st, lpc);
    return;
  }
  if (vw == 1) launch_vw<1, NB_ROWS>(s, comp, fwd, nslot, st, lpc);
  else if (vw == 2) launch_vw<2, NB_ROWS>(s, comp, fwd, nslot, st, lpc);
  else launch_vw<4, NB_ROWS>(s, comp, fwd, nslot, st, lpc);
}

}  // namespace csem
