// complex128 component sweeps of LU-SGS and A-phi as lockstep row pipelines: one launch
// per sweep, the reference's bits.
//
// A sweep updates one field component in the reference's lexicographic Gauss-Seidel order
// (fdfd.c:347-503). In the coupled plane (row r, march m) a point depends on (r-1, m) and
// (r, m-1) (forward; r+1 and m+1 backward); the third axis is independent:
//   Ex: rows k, march j, lines i    Ey: rows k, march i, lines j    Ez: rows j, march i, lines k
// One CTA owns one line of one system and gives every row two threads (one above 256 rows). One
// takes the steps: rows advance in lockstep, skewed by one step per row, and a row's value
// reaches the next row by a warp shuffle or a hand-over between warps. The other makes, a step
// ahead, what the step takes that no row writes during the sweep, and leaves it in shared memory.
//
// The reference's update (fdfd.c:358-369, 384-395, 410-421; own = 0 at the point) is, for
// the three components alike,
//   L_a = ((p0 - up/ds) - (p1 + lo/dsm)) / d   for the march axis and for the row axis,
//   v   = (b - (L_march + L_row) iwmu) / (gg iwmu - sigma)
// with up and lo the component's neighbours along the axis, ds, dsm, d its spacings, and
// p0, p1 the coupling to another component on the point's upper and lower side,
// (A - B) / (line spacing). Written so, every addition, product and quotient is one of the
// reference's up to the signs of its operands, which rounding to nearest respects, so the
// results are its results bit for bit (zeros may differ in sign).
//
// What bounds it is the FP64 unit: 2 operations per SM and cycle. The reference's division
// in every term costs 7 of them, 20 for a zero numerator. Here
//   - divisions run on the integer units (exact_div.h), none of them on the FP64 unit;
//   - gg iwmu depends on (row, march) only and comes with its reciprocal from a table that
//     k_diag64 fills once per application; gg's parts per axis come from the host;
//   - products with iwmu, whose real part is zero, take 2 multiplications instead of 6
//     operations, and p0 of a step is p1 of its neighbour step, kept in registers;
//   - everything that no other row writes during the sweep (p0, p1, lo/dsm, Smith's ratio
//     and denominator) is formed one step ahead, off the dependent chain, by other warps: 1000
//     to 3700 cycles of a step next to the 2700 to 3500 of the chain, instead of after them.
// A point whose operands leave exact_div.h's range (subnormal, infinite, NaN), or any point
// where iwmu has a real part, takes the reference's operations as they stand (slow_point).
// 120 x 120 x 120 cells, one system: 2.95 ms an application; 3.9 ms with one thread a row and the
// FP64 unit's reciprocal of the denominator, 20.0 ms with its divisions (1.54, 1.85 and 9.7 ms
// each where three systems' applications overlap). 128 registers let two lines onto an SM; with
// up to 204 one system takes 2.71 ms, but three 2.15 each.
#include "csem_cuda.cuh"
#include "engine.h"
#include "exact_div.h"
#include "k_sweep_common.cuh"

namespace csem {

using namespace sweep;

namespace {

typedef double2 C;

// a spacing with the reciprocal word of exact_div.h
struct Sp {
  double d;
  uint64_t R;
};
__device__ __forceinline__ Sp sp(const double* d, const uint64_t* q, int n)
{
  Sp s;
  s.d = ro(d + n);
  s.R = q ? (uint64_t)__ldg((const unsigned long long*)q + n) : 0;
  return s;
}
__device__ __forceinline__ C over(C a, Sp s, uint32_t& bad)
{
  return make_double2(xd_div(a.x, s.d, s.R, bad), xd_div(a.y, s.d, s.R, bad));
}

// one axis at one index: ds(n), ds(n-1), d(n)
struct Ax64 {
  Sp s, sm, c;
};
__device__ __forceinline__ Ax64 ax64(const double* d, const double* ds, const uint64_t* q, const uint64_t* qs, int n)
{
  Ax64 a;
  a.s = sp(ds, qs, n);
  a.sm = sp(ds, qs, n - 1);
  a.c = sp(d, q, n);
  return a;
}

// the point by the reference's own operations: neighbours along march and row axis, the
// other components' values A..D on either side, and e = sigma grad v of A-phi
struct Raw {
  C up, lo, A, B, Cc, D;
};
__device__ __noinline__ C slow_point(const Raw& m, const Raw& r, double line_ds, double ms, double msm, double md,
                                     double rs, double rsm, double rd, double gg, double sg, double vol, int fvm,
                                     C b, C e, C iwmu, C iom)
{
  auto L = [&](const Raw& q, double s, double sm, double d) {
    const C t1 = csub<F64>(cdivr<F64>(csub<F64>(q.A, q.B), line_ds), cdivr<F64>(q.up, s));
    const C t2 = cadd<F64>(cdivr<F64>(csub<F64>(q.Cc, q.D), line_ds), cdivr<F64>(q.lo, sm));
    return cdivr<F64>(csub<F64>(t1, t2), d);
  };
  C aij = csub<F64>(cmul<F64>(cadd<F64>(L(m, ms, msm, md), L(r, rs, rsm, rd)), iwmu), e);
  C aii = rmul<F64>(gg, iwmu);
  aii.x = F64::sub(aii.x, sg);
  if (fvm) {
    const C f = rmul<F64>(vol, iom);
    aij = cmul<F64>(aij, f);
    aii = cmul<F64>(aii, f);
  }
  return cdiv<F64>(csub<F64>(b, aij), aii);
}

// A row of a line (r along the row axis): pointers to its own component, the lower row, and the
// coupled components on the upper (A) and lower (B) side of the line, for the march axis (m*)
// and, at this row and the lower one, for the row axis (r*); and its spacings
template <int COMP, bool PHI> struct Row {
  C* own;
  const C *low, *mA, *mB, *rA, *rB, *rC, *rD, *bb, *v1 = nullptr, *v0 = nullptr;  // v: node potential at the edge's two ends
  const double* sg0;
  Sp ln;
  Ax64 Ra;
  __device__ __forceinline__ Row(const SweepP<F64>& s, int slot, int sys, int line, int r)
  {
    const GridP<F64>& g = s.g;
    const int n1 = g.n1, n2 = g.n2;
    const View<F64> V = view_of<F64>(s, slot, sys);
    const int k = COMP == 2 ? line : r, j = COMP == 0 ? 0 : (COMP == 1 ? line : r), i0 = COMP == 0 ? line : 0;
    ln = COMP == 0 ? sp(g.d1s, g.q1s, line) : (COMP == 1 ? sp(g.d2s, g.q2s, line) : sp(g.d3s, g.q3s, line));
    Ra = COMP == 2 ? ax64(g.d2, g.d2s, g.q2, g.q2s, r) : ax64(g.d3, g.d3s, g.q3, g.q3s, r);
    own = V.row(COMP, k, j) + i0;
    low = COMP == 2 ? V.row(2, k, j - 1) : V.row(COMP, k - 1, j) + i0;
    if (COMP == 0) {
      mB = V.row(1, k, 0) + i0, mA = mB + 1;
      rB = V.row(2, k, 0) + i0, rA = rB + 1;
      rD = V.row(2, k - 1, 0) + i0, rC = rD + 1;
    } else if (COMP == 1) {
      mA = V.row(0, k, j + 1), mB = V.row(0, k, j);
      rA = V.row(2, k, j + 1), rB = V.row(2, k, j);
      rC = V.row(2, k - 1, j + 1), rD = V.row(2, k - 1, j);
    } else {
      mA = V.row(0, k + 1, j), mB = V.row(0, k, j);
      rA = V.row(1, k + 1, j), rB = V.row(1, k, j);
      rC = V.row(1, k + 1, j - 1), rD = V.row(1, k, j - 1);
    }
    bb = V.brow(COMP, k, j);
    if (bb) bb += i0;
    sg0 = COMP == 0 ? g.s11 + ix1(n1, n2, k, 0, i0)
                    : (COMP == 1 ? g.s22 + ix2(n1, n2, k, j, 0) : g.s33 + ix3(n1, n2, k, j, 0));
    if (PHI) {
      const C* vp = s.V + (size_t)slot * s.lv;
      v0 = vp + ix3(n1, n2, k, j, i0);
      v1 = COMP == 0 ? v0 + 1 : (COMP == 1 ? vp + ix3(n1, n2, k, j + 1, 0) : vp + ix3(n1, n2, k + 1, j, 0));
    }
  }
  // spacings of the march axis at position m, and the cell volume (Ex's for all three
  // components, fdfd.c:365,391,417)
  static __device__ __forceinline__ Ax64 march(const GridP<F64>& g, int m)
  {
    return COMP == 0 ? ax64(g.d2, g.d2s, g.q2, g.q2s, m) : ax64(g.d1, g.d1s, g.q1, g.q1s, m);
  }
  __device__ __forceinline__ double volume(const GridP<F64>& g, int line, const Ax64& Ma) const
  {
    const double xs = COMP == 0 ? ln.d : Ma.s.d;
    const double yd = COMP == 0 ? Ma.c.d : (COMP == 1 ? ro(g.d2 + line) : Ra.c.d);
    return F64::mul(F64::mul(xs, yd), COMP == 2 ? ro(g.d3 + line) : Ra.c.d);
  }
};

// the whole point (row r, march position m) again by the reference's operations
template <int COMP, bool FWD, bool PHI>
__device__ __noinline__ C slow_row(const SweepP<F64>& s, int slot, int sys, int line, int r, int m_, C prev, C nb)
{
  constexpr bool HASM = COMP != 0 || !FWD, HASR = COMP == 2 || !FWD;
  const GridP<F64>& g = s.g;
  const Row<COMP, PHI> W(s, slot, sys, line, r);
  const SysScal<F64> sc = s.scal[sys];
  const C z = make_double2(0, 0);
  const long m = m_, so = COMP == 0 ? g.n1 : 1, sm = COMP == 0 ? g.n1 + 1 : 1;
  Raw qm{FWD ? z : prev, FWD ? prev : W.own[(m - 1) * so], z, z, z, z};
  Raw qr{FWD ? z : nb, FWD ? nb : W.low[m * so], z, z, z, z};
  if (HASM) qm.A = ro(W.mA + m * sm), qm.B = ro(W.mB + m * sm), qm.Cc = ro(W.mA + (m - 1) * sm), qm.D = ro(W.mB + (m - 1) * sm);
  if (HASR) qr.A = ro(W.rA + m * sm), qr.B = ro(W.rB + m * sm), qr.Cc = ro(W.rC + m * sm), qr.D = ro(W.rD + m * sm);
  const double sg = ro(W.sg0 + m * so);
  const C ee = PHI ? rmul<F64>(sg, cdivr<F64>(csub<F64>(ro(W.v1 + m * sm), ro(W.v0 + m * sm)), W.ln.d)) : z;
  const Ax64 A = W.march(g, m_);
  const double gg = F64::add(COMP == 0 ? ro(g.g2 + m) : ro(g.g1 + m), COMP == 2 ? ro(g.g2 + r) : ro(g.g3 + r));
  return slow_point(qm, qr, W.ln.d, A.s.d, A.sm.d, A.c.d, W.Ra.s.d, W.Ra.sm.d, W.Ra.c.d, gg, sg, W.volume(g, line, A),
                    g.fvm, W.bb ? ro(W.bb + m * so) : z, ee, sc.iwmu, sc.iom);
}

// Smith's quotient by aii in two parts: what depends on aii alone, and the rest
struct Den {
  double r;     // the smaller part of aii over the larger
  XdDen q;      // the denominator
  bool ydom;    // |Re aii| < |Im aii|
};
__device__ __forceinline__ C smith(C a, const Den& n, uint32_t& bad)
{
  const double m1 = F64::mul(n.ydom ? a.x : a.y, n.r), m2 = F64::mul(n.ydom ? a.y : a.x, n.r);
  const double x = F64::add(m1, n.ydom ? a.y : a.x);
  const double y = F64::sub(n.ydom ? m2 : a.y, n.ydom ? a.x : m2);
  return make_double2(xd_div2(x, n.q.d, n.q.R, bad), xd_div2(y, n.q.d, n.q.R, bad));
}

}  // namespace

__host__ __device__ inline long diag64_entries(int n1, int n2, int nK)
{
  return (long)(nK + 1) * (n2 + 1) + (long)(nK + 1) * (n1 + 1) + (long)(n2 + 1) * (n1 + 1);
}

// gg Im(iwmu) and its reciprocal word (0: out of range) of every (row, march) of the three
// components: Ex [k][j], Ey [k][i], Ez [j][i], per slot
__global__ void k_diag64(SweepP<F64> s, ulonglong2* T)
{
  const GridP<F64>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK;
  const long e1 = (long)(nK + 1) * (n2 + 1), e2 = e1 + (long)(nK + 1) * (n1 + 1), e3 = diag64_entries(n1, n2, nK);
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= e3) return;
  const int sys = s.sys_list ? s.sys_list[blockIdx.y] : blockIdx.y;
  const long p = q < e1 ? q : (q < e2 ? q - e1 : q - e2);
  const int nb = q < e1 ? n2 : n1, na = q < e2 ? nK : n2;
  const int a = (int)(p / (nb + 1)), b = (int)(p % (nb + 1));
  ulonglong2 t = make_ulonglong2(0, 0);
  if (a >= 1 && a < na && b >= 1 && b < nb) {
    const double ga = q < e2 ? g.g3[a] : g.g2[a], gb = q < e1 ? g.g2[b] : g.g1[b];
    const double ay = F64::mul(F64::add(ga, gb), s.scal[sys].iwmu.y);
    uint32_t bad = 0;
    const XdDen n = xd_den(ay, bad);
    t.x = xd_bits(ay);
    t.y = bad ? 0 : n.R;
  }
  T[(size_t)blockIdx.y * e3 + q] = t;
}

constexpr int TRAY = 11;  // 16-byte fields of a step's operands

// grid (lines, slots). APHI: A-phi's edge sweep, whose backward pass adds sigma grad v
template <int COMP, bool FWD, bool APHI, int MAXR, bool PAIR>
__global__ void __launch_bounds__(PAIR ? 2 * MAXR : MAXR, PAIR && MAXR <= 128 ? 2 : 1)
    k_sweep64(const __grid_constant__ SweepP<F64> s, const ulonglong2* __restrict__ T)
{
  const int slot = blockIdx.y;
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  const GridP<F64>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, nK = s.nK;
  const int line = blockIdx.x;
  const SysScal<F64> sc = s.scal[sys];
  const C z = make_double2(0, 0);
  constexpr bool HASM = COMP != 0 || !FWD;  // the coupling along the march axis is not zero
  constexpr bool HASR = COMP == 2 || !FWD;  // and along the row axis
  constexpr bool PHI = APHI && !FWD;
  const int R_ = COMP == 2 ? n2 - 1 : nK - 1, M = COMP == 0 ? n2 - 1 : n1 - 1;
  const int rows = PAIR ? blockDim.x / 2 : blockDim.x;
  const bool first = PAIR && threadIdx.x >= rows;  // a row's second thread, which makes the step's operands
  const int rr = threadIdx.x - (first ? rows : 0);
  const bool rowok = rr < R_;
  const int r = rowok ? (FWD ? 1 + rr : R_ - rr) : 1;
  const bool fast = g.q1 != nullptr && sc.iwmu.x == 0. && sc.iom.x == 0.;
  const double wy = sc.iwmu.y;

  const Row<COMP, PHI> W(s, slot, sys, line, r);
  const long so = COMP == 0 ? n1 : 1, sm = COMP == 0 ? n1 + 1 : 1;  // strides along the march
  const ulonglong2* tab = T + (size_t)slot * diag64_entries(n1, n2, nK);
  if (COMP == 0) tab += (long)r * (n2 + 1);
  else tab += (long)(nK + 1) * (n2 + 1) + (COMP == 2 ? (long)(nK + 1) * (n1 + 1) : 0) + (long)r * (n1 + 1);
  auto at = [&](int c) { return FWD ? 1 + c : M - c; };

  // operands of the next step
  C lb = z, pA = z, pB = z, qA = z, qB = z, qC = z, qD = z, lom = z, lor = z, va = z, vb = z;
  double lsg = 0;
  ulonglong2 lt = make_ulonglong2(0, 0);
  Ax64 Mn{};
  auto load = [&](int c) {  // nothing read here is written before that step
    const long m = at(c);
    lb = W.bb ? ro(W.bb + m * so) : z;
    lsg = ro(W.sg0 + m * so);
    lt = __ldg(tab + m);
    Mn = W.march(g, (int)m);
    if (HASM) {  // the side that the step before did not have: upper forward, lower backward
      const long o = (FWD ? m : m - 1) * sm;
      pA = ro(W.mA + o);
      pB = ro(W.mB + o);
    }
    if (HASR) {
      const long o = m * sm;
      qA = ro(W.rA + o);
      qB = ro(W.rB + o);
      qC = ro(W.rC + o);
      qD = ro(W.rD + o);
    }
    if (!FWD) {  // the component's own not-yet-swept neighbours
      lom = W.own[(m - 1) * so];
      lor = W.low[m * so];
    }
    if (PHI) {
      va = ro(W.v1 + m * sm);
      vb = ro(W.v0 + m * sm);
    }
  };
  // what the step takes from them: u = p0 (minus nothing yet), w = p1 + lo/dsm per axis
  C b = z, e = z, um = z, wm = z, ur = z, wr = z, pk = z;
  uint32_t badp = 0, badk = 0;
  double fy = 0;
  Ax64 Ma{};
  Den den{};
  auto make = [&](int c) {
    badp = 0;
    b = lb;
    Ma = Mn;
    if (HASM) {
      uint32_t bn = 0;
      const C p = over(csub<F64>(pA, pB), W.ln, bn);
      if (c == 0) {
        const long o = (FWD ? (long)at(c) - 1 : (long)at(c)) * sm;
        badk = 0;
        pk = over(csub<F64>(ro(W.mA + o), ro(W.mB + o)), W.ln, badk);
      }
      um = FWD ? p : pk;
      wm = FWD ? pk : p;
      badp |= bn | badk;
      pk = p;
      badk = bn;
    }
    if (HASR) {
      ur = over(csub<F64>(qA, qB), W.ln, badp);
      wr = over(csub<F64>(qC, qD), W.ln, badp);
    }
    if (!FWD) {
      wm = cadd<F64>(wm, over(lom, Ma.sm, badp));
      wr = cadd<F64>(wr, over(lor, W.Ra.sm, badp));
    }
    if (PHI) e = rmul<F64>(lsg, over(csub<F64>(va, vb), W.ln, badp));
    const double ay = xd_double(lt.x);
    double x = -lsg, y = ay;
    if (g.fvm) {
      fy = F64::mul(W.volume(g, line, Ma), sc.iom.y);
      x = -F64::mul(ay, fy);
      y = -F64::mul(lsg, fy);
    } else {
      badp |= lt.y == 0 ? 1u : 0u;
    }
    den.ydom = xd_bits(x) << 1 < xd_bits(y) << 1;  // |x| < |y|
    if (den.ydom && !g.fvm) {
      den.r = xd_div2(x, ay, lt.y, badp);
    } else {
      const XdDen n = xd_den(den.ydom ? y : x, badp);
      den.r = xd_div2(den.ydom ? x : y, n.d, n.R, badp);
    }
    den.q = xd_den(F64::add(F64::mul(den.ydom ? x : y, den.r), den.ydom ? y : x), badp);
  };
  // one step of a row: prev is its value at the march position before, nb the row before's at
  // this one
  auto step = [&](int c, C prev, C nb) {
    uint32_t bad = fast ? badp : 1u;
    C v = z;
    if (fast) {  // (both axes at a time: their chains are as long)
      const C em = over(prev, FWD ? Ma.sm : Ma.s, bad), er = over(nb, FWD ? W.Ra.sm : W.Ra.s, bad);
      const C Lm = over(FWD ? csub<F64>(um, cadd<F64>(wm, em)) : csub<F64>(csub<F64>(um, em), wm), Ma.c, bad);
      const C Lr = over(FWD ? csub<F64>(ur, cadd<F64>(wr, er)) : csub<F64>(csub<F64>(ur, er), wr), W.Ra.c, bad);
      const C S = cadd<F64>(Lm, Lr);
      C a = make_double2(-F64::mul(S.y, wy), F64::mul(S.x, wy));
      if (PHI) a = csub<F64>(a, e);
      if (g.fvm) a = make_double2(-F64::mul(a.y, fy), F64::mul(a.x, fy));
      v = smith(csub<F64>(b, a), den, bad);
    }
    if (bad) v = slow_row<COMP, FWD, PHI>(s, slot, sys, line, r, at(c), prev, nb);
    W.own[(long)at(c) * so] = v;
    return v;
  };
  const int steps = M + R_ - 1;
  if constexpr (PAIR) {
    extern __shared__ ulonglong2 smem[];
    // a step's operands, [parity][field][row], and the last rows of the warps, [parity][warp]
    ulonglong2* const tray = smem + rr;
    C* const last = (C*)(smem + 2 * TRAY * rows);
    const int lane = threadIdx.x & 31, w = rr >> 5, nw = rows >> 5;
    // up to 4 warps hand over by named barriers (1 .. 6) and meet their second warps at 7 .. 10
    constexpr bool NAMED = MAXR <= 128;
    auto meet = [&]() {
      if constexpr (NAMED) nbar_sync(7 + w);
      else __syncthreads();
    };
    auto put = [&](ulonglong2*& p, double x, double y) {
      *p = make_ulonglong2(xd_bits(x), xd_bits(y));
      p += rows;
    };
    auto take = [&](const ulonglong2*& p) {
      const ulonglong2 u = *p;
      p += rows;
      return make_double2(xd_double(u.x), xd_double(u.y));
    };
    if (first) {
      if (fast && rowok && rr == 0 && M > 0) load(0);
      for (int t = -1; t < steps; t++) {
        const int c = t + 1 - rr;
        if (fast && rowok && c >= 0 && c < M) {
          make(c);
          ulonglong2* p = tray + (t + 1 & 1) * TRAY * rows;
          put(p, b.x, b.y);
          if (HASM || !FWD) put(p, um.x, um.y), put(p, wm.x, wm.y);
          if (HASR || !FWD) put(p, ur.x, ur.y), put(p, wr.x, wr.y);
          if (PHI) put(p, e.x, e.y);
          const Sp msp = FWD ? Ma.sm : Ma.s;
          put(p, msp.d, xd_double(msp.R));
          put(p, Ma.c.d, xd_double(Ma.c.R));
          put(p, den.r, den.q.d);
          put(p, xd_double(den.q.R), xd_double((badp ? 1u : 0u) | (den.ydom ? 2u : 0u)));
          if (g.fvm) put(p, fy, 0.);
        }
        if (fast && rowok && c + 1 >= 0 && c + 1 < M) load(c + 1);
        meet();
      }
      return;
    }
    C res = z;
    meet();
    for (int t = 0; t < steps; t++) {
      const int c = t - rr;
      C nb = make_double2(__shfl_up_sync(0xffffffffu, res.x, 1), __shfl_up_sync(0xffffffffu, res.y, 1));
      const bool wait = NAMED && w > 0 && t > 0;
      if (wait) nbar_sync(2 * w - 1);  // the warp before has written step t - 1
      if (lane == 0) nb = w > 0 && t > 0 ? last[(NAMED ? 0 : (t - 1 & 1) * nw) + w - 1] : z;
      if (wait) nbar_arrive(2 * w);  // and may write step t
      if (rowok && c >= 0 && c < M) {
        if (fast) {
          const ulonglong2* p = tray + (t & 1) * TRAY * rows;
          b = take(p);
          if (HASM || !FWD) um = take(p), wm = take(p);
          if (HASR || !FWD) ur = take(p), wr = take(p);
          if (PHI) e = take(p);
          C q = take(p);
          (FWD ? Ma.sm : Ma.s).d = q.x, (FWD ? Ma.sm : Ma.s).R = xd_bits(q.y);
          q = take(p);
          Ma.c.d = q.x, Ma.c.R = xd_bits(q.y);
          q = take(p);
          den.r = q.x, den.q.d = q.y;
          q = take(p);
          den.q.R = xd_bits(q.x);
          badp = (uint32_t)xd_bits(q.y) & 1, den.ydom = (xd_bits(q.y) & 2) != 0;
          if (g.fvm) fy = take(p).x;
        }
        res = step(c, c > 0 ? res : z, nb);
      } else {
        res = z;
      }
      const bool next = NAMED && w + 1 < nw;
      if (next && t > 0) nbar_sync(2 * w + 2);  // the next warp has read step t - 1
      if (lane == 31) last[(NAMED ? 0 : (t & 1) * nw) + w] = res;
      if (next) nbar_arrive(2 * w + 1);
      meet();
    }
    if (NAMED && w > 0 && steps > 0) nbar_sync(2 * w - 1);  // the barriers' last generation
  } else {
    __shared__ HandOff<1, C, (MAXR <= NB_ROWS)> hand;
    C res[1] = {z};
    if (fast && rowok && rr == 0 && M > 0) {
      load(0);
      make(0);
    }
    for (int t = 0; t < steps; t++) {
      const int c = t - rr;
      const bool act = rowok && c >= 0 && c < M;
      const bool nxt = fast && rowok && c + 1 >= 0 && c + 1 < M;
      if (nxt) load(c + 1);
      C nb[1];
      hand.get(res, nb, t);
      res[0] = act ? step(c, c > 0 ? res[0] : z, nb[0]) : z;
      hand.put(res, t);
      if (nxt) make(c + 1);
    }
    hand.finish(steps);
  }
}

// One hyperplane i + j + k = t of A-phi's node sweep (fdfd.c:654-710), as k_aphi_phi with
// quotients on the integer units: of its 29 divisions per node the node's own diagonal is a sum of
// host-made terms, and the others take no FP64 operation. A node where a quotient is out of range
// is done again with the / operator. What is left is bound by latency, at some 6 us a hyperplane
// (84^3 cells: 17 with the divisions; 474 hyperplanes an application, which takes 5.2 ms instead
// of 10.7, 2.4 instead of 4.4 where three overlap; and 4.3 and 2.1 with a hyperplane's blocks
// started, and what does not depend on it loaded, while the one before still runs).
template <bool FWD>
__global__ void __launch_bounds__(128) k_aphi_phi64(const __grid_constant__ SweepP<F64> s, C* __restrict__ VV, int t)
{
  const int slot = blockIdx.z;
  const GridP<F64>& g = s.g;
  const int n1 = g.n1, n2 = g.n2, n3 = g.n3;
  const int i = 1 + blockIdx.x * 32 + threadIdx.x, j = 1 + blockIdx.y * 4 + threadIdx.y, k = t - i - j;
  cudaTriggerProgrammaticLaunchCompletion();  // the next hyperplane's blocks may come in and wait
  if (i >= n1 || j >= n2 || k < 1 || k >= n3) return;
  const int sys = s.sys_list ? s.sys_list[slot] : slot;
  C* v = VV + (size_t)slot * s.lv;
  const long q = ix3(n1, n2, k, j, i), qj = ix3(n1, n2, k, j - 1, i), qk = ix3(n1, n2, k - 1, j, i);
  const C* ax = s.Y + (size_t)sys * g.lE;
  const C *ay = ax + g.lEx, *az = ay + g.lEy;
  const C z = make_double2(0, 0);
  const Ax64 X = ax64(g.d1, g.d1s, g.q1, g.q1s, i), Y = ax64(g.d2, g.d2s, g.q2, g.q2s, j), Z = ax64(g.d3, g.d3s, g.q3, g.q3s, k);
  const double geo = F64::add(F64::add(ro(g.g1 + i), ro(g.g2 + j)), ro(g.g3 + k));
  const C b = ro(s.BV + (size_t)slot * s.lv + q);
  const SysScal<F64> sc = s.scal[sys];
  // everything but v is older than the sweep's first launch: read it before waiting for the
  // hyperplane before (which some block of every hyperplane does, so they end in order)
  const double s1p = ro(g.s11 + ix1(n1, n2, k, j, i)), s1m = ro(s.s11u + ix1(n1, n2, k, j, i - 1));
  const double s2p = ro(g.s22 + ix2(n1, n2, k, j, i)), s2m = ro(s.s22u + ix2(n1, n2, k, j - 1, i));
  const double s3p = ro(g.s33 + ix3(n1, n2, k, j, i)), s3m = ro(s.s33u + ix3(n1, n2, k - 1, j, i));
  const C a1p = ro(ax + ix1(n1, n2, k, j, i)), a1m = ro(ax + ix1(n1, n2, k, j, i - 1));
  const C a2p = ro(ay + ix2(n1, n2, k, j, i)), a2m = ro(ay + ix2(n1, n2, k, j - 1, i));
  const C a3p = ro(az + ix3(n1, n2, k, j, i)), a3m = ro(az + ix3(n1, n2, k - 1, j, i));
  uint32_t bad = 0;
  const XdDen den = xd_den(-geo, bad);
  cudaGridDependencySynchronize();
  auto node = [&](auto over_) {
    // sigma (a + (hi - lo) / ds) on a face; v is zero at the node itself
    auto face = [&](double sg, C a, C dv, Sp ds) { return rmul<F64>(sg, cadd<F64>(a, over_(dv, ds))); };
    auto axis = [&](C up, C lo, double sp, double sm, C ap, C am, const Ax64& A) {
      return over_(csub<F64>(face(sp, ap, up, A.s), face(sm, am, csub<F64>(z, lo), A.sm)), A.c);
    };
    const C x = axis(FWD ? z : v[ix3(n1, n2, k, j, i + 1)], v[q - 1], s1p, s1m, a1p, a1m, X);
    const C y = axis(FWD ? z : v[ix3(n1, n2, k, j + 1, i)], v[qj], s2p, s2m, a2p, a2m, Y);
    const C w = axis(FWD ? z : v[ix3(n1, n2, k + 1, j, i)], v[qk], s3p, s3m, a3p, a3m, Z);
    return cadd<F64>(cadd<F64>(x, y), w);
  };
  C aij = node([&](C a, Sp d) { return over(a, d, bad); });
  C r = z;
  if (!g.fvm) {
    const C a = csub<F64>(b, aij);
    r = make_double2(xd_div2(a.x, den.d, den.R, bad), xd_div2(a.y, den.d, den.R, bad));
  }
  if (bad || g.fvm) {
    if (bad) aij = node([&](C a, Sp d) { return cdivr<F64>(a, d.d); });
    C aii = make_double2(-geo, 0);
    if (g.fvm) {
      const C f = rmul<F64>(F64::mul(F64::mul(X.s.d, Y.c.d), Z.c.d), sc.iom);
      aij = cmul<F64>(aij, f);
      aii = cmul<F64>(aii, f);
    }
    r = cdiv<F64>(csub<F64>(b, aij), aii);
  }
  v[q] = r;
}

void launch_aphi_phi64(const SweepP<F64>& s, double2* V, int t, int nslot, cudaStream_t st)
{
  const PlaneLaunch L(s, t, nslot, st);
  count_launch();
  if (t > 0) cudaLaunchKernelEx(&L.cfg, k_aphi_phi64<true>, s, V, t);
  else cudaLaunchKernelEx(&L.cfg, k_aphi_phi64<false>, s, V, -t);
}

template <int COMP, bool FWD, bool APHI>
static void launch64(const SweepP<F64>& s, int nslot, const ulonglong2* T, cudaStream_t st)
{
  const int rows = COMP == 2 ? s.g.n2 - 1 : s.nK - 1;
  const int threads = (rows + 31) / 32 * 32;
  dim3 grd(COMP == 0 ? s.g.n1 : (COMP == 1 ? s.g.n2 : s.nK), nslot);
  // two threads a row while a CTA can hold them
  const size_t sm = (size_t)threads * 2 * TRAY * 16 + 2 * (threads / 32) * 16;
  count_launch();
  if (rows > NB_ROWS) {
    k_sweep64<COMP, FWD, APHI, MAXROWS, false><<<grd, threads, 0, st>>>(s, T);
  } else if (rows > 128) {
    allow_smem<k_sweep64<COMP, FWD, APHI, NB_ROWS, true>>(sm);
    k_sweep64<COMP, FWD, APHI, NB_ROWS, true><<<grd, 2 * threads, sm, st>>>(s, T);
  } else {
    allow_smem<k_sweep64<COMP, FWD, APHI, 128, true>>(sm);
    k_sweep64<COMP, FWD, APHI, 128, true><<<grd, 2 * threads, sm, st>>>(s, T);
  }
}

size_t sweep64_table_bytes(int n1, int n2, int nK) { return sizeof(ulonglong2) * (size_t)diag64_entries(n1, n2, nK); }

void launch_sweep64_table(const SweepP<F64>& s, int nslot, void* T, cudaStream_t st)
{
  const long n = diag64_entries(s.g.n1, s.g.n2, s.nK);
  dim3 grd((unsigned)((n + 127) / 128), nslot);
  count_launch(), k_diag64<<<grd, 128, 0, st>>>(s, (ulonglong2*)T);
}

void launch_sweep64(const SweepP<F64>& s, int comp, bool fwd, bool aphi, int nslot, const void* Tv, cudaStream_t st)
{
  const ulonglong2* T = (const ulonglong2*)Tv;
  // (A-phi's forward edge sweeps are LU-SGS's)
  if (comp == 0) {
    if (fwd) launch64<0, true, false>(s, nslot, T, st);
    else if (aphi) launch64<0, false, true>(s, nslot, T, st);
    else launch64<0, false, false>(s, nslot, T, st);
  } else if (comp == 1) {
    if (fwd) launch64<1, true, false>(s, nslot, T, st);
    else if (aphi) launch64<1, false, true>(s, nslot, T, st);
    else launch64<1, false, false>(s, nslot, T, st);
  } else {
    if (fwd) launch64<2, true, false>(s, nslot, T, st);
    else if (aphi) launch64<2, false, true>(s, nslot, T, st);
    else launch64<2, false, false>(s, nslot, T, st);
  }
}

}  // namespace csem
