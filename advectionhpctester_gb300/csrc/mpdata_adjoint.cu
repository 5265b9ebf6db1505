// Adjoint of the MPDATA step (infinite-gauge and standard forms, iord >= 2
// corrective passes, nonoscillatory limiter on or off).  No reference code exists for
// it; it differentiates the forward step of mpdata_body.cuh exactly, with
// every branch (pp, pn, min3, the limiter's max/min over the 7-point stars
// and over the running extrema of earlier passes, abs) taken at the forward
// values ("piecewise at the forward branch").
//
// Given psi at the start of a step, the velocities and lambda = dJ/dpsi_new,
// the step adjoint first records the forward step pass by pass (upwind field,
// face reciprocals; per pass its input field, pseudo-velocities, limiter
// ratios, limited velocities and running extrema), then runs one reverse
// kernel per forward stage, last pass first:
//   update    x_out = rhr*(q - div(w)/h)           -> lambda_x, lambda_w
//             (standard: rhr*(q - div(g)*hinv), g the limited donor fluxes of q)
//   limiter   w = pp(v)*A1 - pn(v)*A2              -> lambda_v, lambda_cp, lambda_cn
//             (standard: the sign-aware vlim_std and g = donor(q, w))
//   bounds    cp,cn from the extrema and v         -> lambda_x, lambda_v, and lambda of
//                                                     the step input (first pass) or of
//                                                     the previous pass's extrema
//   pseudo    v(x, a)                              -> lambda_x, and lambda_a: the
//                                                     velocity gradient (first pass) or
//                                                     the previous pass's lambda_w
//   upwind    xant(psi, u)                         -> lambda_psi, lambda_u
// Each reverse kernel walks the forward stage's reads (with the same boundary
// index maps), so wall faces (constant zero), mirrored z faces and periodic
// wraps are transposed exactly as the forward reads them.  What belongs to the
// cell or to a face it owns is stored; the rest is scattered with atomic adds
// (the bounds, the pseudo-velocity in FP64 and at walls) or gathered.  The
// summation order of the atomics is not fixed: results agree with the FP64
// AD oracle to rounding, not bit for bit.
// Gauge form, per field of 256x256x64 FP64 cells (33 MB): clearing all 19
// accumulators took 95 us of a step adjoint; only those that the first kernel
// to touch them adds to are cleared now (lcp and lcn at iord 2).
#include "mpdata_body.cuh"
#include "mpdata_stages.cuh"

namespace mpdata {

// Launch bounds of the reverse kernels: minimum resident 128-thread blocks
// per SM (0: no explicit bound).  Build-time overridable for tuning sweeps;
// a sweep of 6-16 blocks per kernel measured within 0.5% of no bound.
#ifndef MPDATA_MINB_KA_PSEUDO
#define MPDATA_MINB_KA_PSEUDO 0
#endif
#ifndef MPDATA_MINB_KA_BOUNDS
#define MPDATA_MINB_KA_BOUNDS 0
#endif
#ifndef MPDATA_MINB_KA_UPWIND
#define MPDATA_MINB_KA_UPWIND 0
#endif
#ifndef MPDATA_MINB_KA_LIMIT
#define MPDATA_MINB_KA_LIMIT 0
#endif
#ifndef MPDATA_MINB_KA_UPDATE
#define MPDATA_MINB_KA_UPDATE 0
#endif
#define KA_BOUND_(n) __launch_bounds__(128, n)
#define KA_BOUND0 __launch_bounds__(128)
#if MPDATA_MINB_KA_PSEUDO > 0
#define KA_LB_PSEUDO KA_BOUND_(MPDATA_MINB_KA_PSEUDO)
#else
#define KA_LB_PSEUDO KA_BOUND0
#endif
#if MPDATA_MINB_KA_BOUNDS > 0
#define KA_LB_BOUNDS KA_BOUND_(MPDATA_MINB_KA_BOUNDS)
#else
#define KA_LB_BOUNDS KA_BOUND0
#endif
#if MPDATA_MINB_KA_UPWIND > 0
#define KA_LB_UPWIND KA_BOUND_(MPDATA_MINB_KA_UPWIND)
#else
#define KA_LB_UPWIND KA_BOUND0
#endif
#if MPDATA_MINB_KA_LIMIT > 0
#define KA_LB_LIMIT KA_BOUND_(MPDATA_MINB_KA_LIMIT)
#else
#define KA_LB_LIMIT KA_BOUND0
#endif
#if MPDATA_MINB_KA_UPDATE > 0
#define KA_LB_UPDATE KA_BOUND_(MPDATA_MINB_KA_UPDATE)
#else
#define KA_LB_UPDATE KA_BOUND0
#endif
// The record kernels run the forward stage bodies: the forward stage
// kernels' bounds (FP64 / FP32).
template <class R, int N64, int N32>
struct KfMinBlocks {
  static constexpr int v = sizeof(R) == 8 ? N64 : N32;
};

// ---- adjoints of the read maps --------------------------------------------
// Adding a zero changes no accumulator (they start at +0), so zero
// contributions, frequent where the limiter is inactive, skip the atomic; the
// test is an integer one on the FP64 bit pattern.
__device__ __forceinline__ bool nonzero(double v) { return nonzero_bits(v); }
__device__ __forceinline__ bool nonzero(float v) { return v != 0.0f; }
template <class R>
__device__ __forceinline__ void addat(const Arr<R>& A, int i, int j, int k, R v) {
  if (nonzero(v)) atomicAdd(&A.at(i, j, k), v);
}
// xr(): the field with the xant halo rule (reflection or wrap).  IN: the
// index is inside the grid (a cell in [2, n-1] reading +-1), the map is the
// identity.
template <class R, bool IN = false>
__device__ __forceinline__ void xr_add(const Geo& g, const Arr<R>& L, int i, int j, int k, R v) {
  if (IN) { addat(L, i, j, k, v); return; }
  addat(L, g.bx ? wrapi(i, g.np) : refl(i, g.np), g.by ? wrapi(j, g.mp) : refl(j, g.mp), cz(g, k), v);
}
// fx/fy/fz<AIN>()
template <class R, bool AIN, bool IN = false>
__device__ __forceinline__ void fx_add(const Geo& g, const Arr<R>& A, int f, int j, int k, R v) {
  if (IN) { addat(A, f, j, k, v); return; }
  j = cy(g, j);
  k = cz(g, k);
  if (g.bx) { addat(A, wrapi(f, g.np), j, k, v); return; }
  if (AIN) { addat(A, f, j, k, v); return; }
  if (f <= 1 || f > g.np) return;  // wall faces are the constant 0
  addat(A, f, j, k, v);
}
template <class R, bool AIN, bool IN = false>
__device__ __forceinline__ void fy_add(const Geo& g, const Arr<R>& A, int i, int f, int k, R v) {
  if (IN) { addat(A, i, f, k, v); return; }
  i = cx(g, i);
  k = cz(g, k);
  if (g.by) { addat(A, i, wrapi(f, g.mp), k, v); return; }
  if (AIN) { addat(A, i, f, k, v); return; }
  if (f <= 1 || f > g.mp) return;
  addat(A, i, f, k, v);
}
template <class R, bool AIN, bool IN = false>
__device__ __forceinline__ void fz_add(const Geo& g, const Arr<R>& A, int i, int j, int f, R v) {
  if (IN) { addat(A, i, j, f, v); return; }
  i = cx(g, i);
  j = cy(g, j);
  if (g.bz) { addat(A, i, j, wrapi(f, g.lp), v); return; }
  if (AIN) { addat(A, i, j, f, v); return; }
  if (f <= 1) { addat(A, i, j, 2, -v); return; }       // face 1 reads -face 2
  if (f > g.lp) { addat(A, i, j, g.lp, -v); return; }  // face lp+1 reads -face lp
  addat(A, i, j, f, v);
}

// derivative conventions of the branches (forward values decide); the
// tests are integer ones on the sign bit and the magnitude bits
template <class R> __device__ __forceinline__ R dpp(R y) { return (!sgn(y) && nonzero(y)) ? R(1) : R(0); }
template <class R> __device__ __forceinline__ R dpn(R y) { return (sgn(y) && nonzero(y)) ? R(-1) : R(0); }
template <class R> __device__ __forceinline__ R dabs(R y) { return sgn(y) ? R(-1) : R(1); }


template <class R> __device__ __forceinline__ R negv(R x) { return -x; }
template <> __device__ __forceinline__ double negv<double>(double x) { return neg_bits(x); }
__device__ __forceinline__ bool is_one(float v) { return v == 1.0f; }

// Reverse kernels: the body is a device function of (i,j,k) templated on
// IN; warps away from every wall take IN = true.
#define ADISPATCH(CALL)                                      \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;  \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;  \
  const int k = blockIdx.z + 1;                              \
  const bool win = warp_interior(P.g, i, j, k);              \
  if (i > P.g.np || j > P.g.mp) return;                      \
  if (win) {                                                 \
    CALL(true);                                              \
  } else {                                                   \
    CALL(false);                                             \
  }

#define ACELL                                                \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;  \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;  \
  const int k = blockIdx.z + 1;                              \
  if (i > P.g.np || j > P.g.mp) return;                      \
  const Geo& g = P.g;

// The workspace's fields have one layout: a cell is one offset in all of them.
template <class R>
struct Nbr {  // offset of a cell and differences to its neighbours, wrapped
  long o;
  int xm, xp, ym, yp;
  long zm, zp;
  __device__ __forceinline__ Nbr(const Geo& g, const Arr<R>& A, int i, int j, int k) {
    o = A.off(i, j, k);
    xm = i > 1 ? -1 : g.np - 1;
    xp = i < g.np ? 1 : 1 - g.np;
    ym = j > 1 ? -A.sy : (g.mp - 1) * A.sy;
    yp = j < g.mp ? A.sy : (1 - g.mp) * A.sy;
    zm = k > 1 ? -(long)A.sz : (long)(g.lp - 1) * A.sz;
    zp = k < g.lp ? (long)A.sz : (long)(1 - g.lp) * A.sz;
  }
};
// ---- update: x_new = rhr*(q - D/h), D = sum of signed limited fluxes -------
// The adjoint of D is one value per cell (lq); the limiter's reverse takes a
// face's lambda_w from the two cells it separates, so nothing is scattered.
// After the last pass's read of the caller's lambda (A.lx set), that array
// becomes the accumulator of the step input's adjoint.  256x256x64 FP64: 31 us,
// at the rate of its five fields; six atomics a cell took 61.
template <class R>
__global__ void KA_LB_UPDATE ka_update(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  const bool in = i <= P.g.np && j <= P.g.mp;
  const unsigned act = __ballot_sync(0xffffffffu, in);
  if (!in) return;
  const R ln = A.lam.ld(i, j, k);
  const R rh = P.rhr.ld(i, j, k), h = P.h.ld(i, j, k);
  if (A.lx.p) A.lx.at(i, j, k) = R(0);
  if (__all_sync(act, is_one(rh) && is_one(h))) {  // x*1 == x/1 == x
    A.lxant.at(i, j, k) = ln;
    A.lq.at(i, j, k) = negv(ln);
    return;
  }
  const R lt = rh * ln;                 // d x_new / d t, t = q - D/h
  A.lxant.at(i, j, k) = quot(lt, rh);   // q = xant/rhr
  A.lq.at(i, j, k) = quot(-lt, h);
}

// ---- limiter: w = pp(v)*min3(cp(c),cn(c-1)) - pn(v)*min3(cp(c-1),cn(c)) -------
// min3(a,b) = mn2(mn2(1,a),b): b is taken when b <= t, else a when a <= 1.
// The ratios are non-negative (or RATIO_CAP), so for doubles their bit
// patterns order as their values and the compares run on the integer pipe.
__device__ __forceinline__ bool lt_nonneg(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ bool lt_nonneg(float a, float b) { return a < b; }
template <class R> __device__ __forceinline__ bool min3_takes_b(R a, R b) {
  return !lt_nonneg(lt_nonneg(R(1), a) ? R(1) : a, b);
}
template <class R> __device__ __forceinline__ bool min3_takes_a(R a, R b) {
  return !min3_takes_b(a, b) && !lt_nonneg(R(1), a);
}
template <class R>
__device__ __forceinline__ void min3_adj(R a, R b, R lam, const Arr<R>& La, int ia, int ja, int ka,
                                         const Arr<R>& Lb, int ib, int jb, int kb) {
  if (min3_takes_b(a, b)) addat(Lb, ib, jb, kb, lam);
  else if (min3_takes_a(a, b)) addat(La, ia, ja, ka, lam);
}

// A cell owns its lower face on each axis.  The face's lambda_w is lq of the
// cell below minus lq of the cell above; at a z wall the mirrored face doubles
// the wall cell's share of its inner face (exact).  LW, where it is given,
// holds what the next pass (or the density step's mass fluxes) added to
// lambda_w.  lambda_v is stored whole (the bounds' reverse adds to it); only
// the ratios that limit their flux, a minority, are added to by atomics.
template <class R, bool NONOS>
__global__ void KA_LB_LIMIT ka_limit(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  ACELL
  const Nbr<R> n(g, A.lq, i, j, k);
  const long o = n.o, ov = P.v1.off(i, j, k);  // the recorded velocities may lie in a padded arena
  const R *const cp = P.cp.p + o, *const cn = P.cn.p + o, *const lq = A.lq.p + o;
  const R cpc = NONOS ? cp[0] : R(0), cnc = NONOS ? cn[0] : R(0), qc = lq[0];
  auto face = [&](const Arr<R>& V, const Arr<R>& LV, const Arr<R>& LW, long d, R ql, R qr) {
    const R v = V.p[ov];
    R lw = ql - qr;
    if (LW.p) lw += LW.p[o];
    if (!NONOS) {
      LV.p[o] = lw;
      return;
    }
    // dw/dv = a1 (v > 0), a2 (v < 0), 0; dw/da1 = pp(v), dw/da2 = -pn(v): one of
    // them is v, the other zero.  cp is of the cell the flux enters, cn of the
    // one it leaves
    const R cpm = cp[d], cnm = cn[d];
    const bool vz = !nonzero(v), vn = sgn(v);
    const R a = vn ? cpm : cpc, b = vn ? cnc : cnm;
    LV.p[o] = vz ? R(0) : lw * min3(a, b);
    const bool tb = min3_takes_b(a, b), ta = !tb && !lt_nonneg(R(1), a);
    if (!vz && (ta || tb)) atomicAdd((ta ? A.lcp.p : A.lcn.p) + (vn == ta ? o + d : o), lw * v);
  };
  if (g.bx || i > 1) face(P.v1, A.lv1, A.lw1, n.xm, lq[n.xm], qc);
  if (g.by || j > 1) face(P.v2, A.lv2, A.lw2, n.ym, lq[n.ym], qc);
  if (g.bz || k > 1) {
    R ql = lq[n.zm], qr = qc;
    if (!g.bz && k == 2) ql = scale_up<1>(ql);
    if (!g.bz && k == g.lp) qr = scale_up<1>(qr);
    face(P.v3, A.lv3, A.lw3, n.zm, ql, qr);
  }
}

// ---- bounds: cp = (mx-x)h/Dp, cn = (x-mn)h/Dn -------------------------------
// The extrema are re-folded in the oracle's order (mx2/mn2 trees) with the
// compare-and-select's own semantics (ties, +0 == -0 included, keep the
// second operand), so each goes to the same operand: element ids 0..6 are
// x_in, 7..13 xant (centre 1 and 8; the lower and upper neighbours along x, y,
// z at 0, 2, 3, 4, 5, 6 and 7 more).  FP64 values compare on the integer pipe
// (ieee_gt).
__device__ __forceinline__ bool arg_gt(double a, double b) { return ieee_gt(a, b); }
__device__ __forceinline__ bool arg_gt(float a, float b) { return a > b; }
template <class R>
struct Arg {
  R v;
  int id;
};
template <class R> __device__ __forceinline__ Arg<R> mkarg(R v, int id) { return Arg<R>{v, id}; }
template <class R> __device__ __forceinline__ Arg<R> amax(Arg<R> a, Arg<R> b) { return arg_gt(a.v, b.v) ? a : b; }
template <class R> __device__ __forceinline__ Arg<R> amin(Arg<R> a, Arg<R> b) { return arg_gt(b.v, a.v) ? a : b; }

// FIRST: the fold starts from the step input's star (ids 0..6); later passes
// start from the previous pass's running extrema (id 14).  The current
// field's star is ids 7..13.  x_in is read with the zero-gradient map, the
// current field with the reflection map.
template <class R, bool FIRST, bool IN>
struct StarFold {
  int im, ip, jm, jp, km, kp, ri_m, ri_p, rj_m, rj_p;
  Arg<R> ma, mi;
  __device__ __forceinline__ StarFold(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
    const Geo& g = P.g;
    const bool lo = IN || g.bz || k > 1, hi = IN || g.bz || k < g.lp;
    im = IN ? i - 1 : (g.bx ? wrapi(i - 1, g.np) : clampi(i - 1, g.np));
    ip = IN ? i + 1 : (g.bx ? wrapi(i + 1, g.np) : clampi(i + 1, g.np));
    jm = IN ? j - 1 : (g.by ? wrapi(j - 1, g.mp) : clampi(j - 1, g.mp));
    jp = IN ? j + 1 : (g.by ? wrapi(j + 1, g.mp) : clampi(j + 1, g.mp));
    km = cz<IN>(g, k - 1);
    kp = cz<IN>(g, k + 1);
    ri_m = IN ? i - 1 : (g.bx ? wrapi(i - 1, g.np) : refl(i - 1, g.np));
    ri_p = IN ? i + 1 : (g.bx ? wrapi(i + 1, g.np) : refl(i + 1, g.np));
    rj_m = IN ? j - 1 : (g.by ? wrapi(j - 1, g.mp) : refl(j - 1, g.mp));
    rj_p = IN ? j + 1 : (g.by ? wrapi(j + 1, g.mp) : refl(j + 1, g.mp));
    const Arr<R>& X = P.xant;
    const Arr<R>& xin = P.psi;
    if (FIRST) {
      const Arg<R> e0 = mkarg(xin.ld(im, j, k), 0), e1 = mkarg(xin.ld(i, j, k), 1), e2 = mkarg(xin.ld(ip, j, k), 2),
                   e3 = mkarg(xin.ld(i, jm, k), 3), e4 = mkarg(xin.ld(i, jp, k), 4),
                   e5 = mkarg(xin.ld(i, j, km), 5), e6 = mkarg(xin.ld(i, j, kp), 6);
      ma = amax(amax(amax(e0, e1), amax(e2, e3)), e4);
      mi = amin(amin(amin(e0, e1), amin(e2, e3)), e4);
      if (lo) { ma = amax(ma, e5); mi = amin(mi, e5); }
      if (hi) { ma = amax(ma, e6); mi = amin(mi, e6); }
    } else {
      ma = mkarg(A.mxp.ld(i, j, k), 14);
      mi = mkarg(A.mnp.ld(i, j, k), 14);
    }
    const Arg<R> f0 = mkarg(X.ld(ri_m, j, k), 7), f1 = mkarg(X.ld(i, j, k), 8), f2 = mkarg(X.ld(ri_p, j, k), 9),
                 f3 = mkarg(X.ld(i, rj_m, k), 10), f4 = mkarg(X.ld(i, rj_p, k), 11),
                 f5 = mkarg(X.ld(i, j, km), 12), f6 = mkarg(X.ld(i, j, kp), 13);
    ma = amax(amax(amax(ma, f0), amax(f1, f2)), amax(f3, f4));
    mi = amin(amin(amin(mi, f0), amin(f1, f2)), amin(f3, f4));
    if (lo) { ma = amax(ma, f5); mi = amin(mi, f5); }
    if (hi) { ma = amax(ma, f6); mi = amin(mi, f6); }
  }
  // adds v to the adjoint of the element id (not 14)
  __device__ __forceinline__ void add(const AdjArr<R>& A, int id, int i, int j, int k, R v) const {
    const bool in = FIRST && id < 7;
    const int n = in ? id : id - 7;
    const int ii = n == 0 ? (in ? im : ri_m) : n == 2 ? (in ? ip : ri_p) : i;
    const int jj = n == 3 ? (in ? jm : rj_m) : n == 4 ? (in ? jp : rj_p) : j;
    const int kk = n == 5 ? km : n == 6 ? kp : k;
    addat(in ? A.lx : A.lxant, ii, jj, kk, v);
  }
};

// Adjoint of the bounds' denominators onto one flux f: Dp holds pn(f) and
// Dn pp(f) for an outflow face (e), the reverse for an inflow face (w); a
// zero flux contributes to neither.
template <class R>
__device__ __forceinline__ R lflux(R f, R lDp, R lDn, bool inflow) {
  if (!nonzero(f)) return R(0);
  const bool neg = sgn(f);
  if (inflow) return neg ? -lDn : lDp;
  return neg ? -lDp : lDn;
}

// STD: the fluxes of the bounds are the unlimited donor fluxes f*ns (their
// adjoint goes to lf); gauge: the pseudo-velocities themselves (lv).
template <class R, bool FIRST, bool STD, bool IN>
__device__ __forceinline__ void ka_bounds_cell(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
  const Geo& g = P.g;
  const StarFold<R, FIRST, IN> x(P, A, i, j, k);
  const Arr<R>& F1 = STD ? P.f1 : P.v1;
  const Arr<R>& F2 = STD ? P.f2 : P.v2;
  const Arr<R>& F3 = STD ? P.f3 : P.v3;
  const Arr<R>& LF1 = STD ? A.lf1 : A.lv1;
  const Arr<R>& LF2 = STD ? A.lf2 : A.lv2;
  const Arr<R>& LF3 = STD ? A.lf3 : A.lv3;
  const R e1 = fx<R, false, IN>(g, F1, i + 1, j, k), w1 = fx<R, false, IN>(g, F1, i, j, k);
  const R e2 = fy<R, false, IN>(g, F2, i, j + 1, k), w2 = fy<R, false, IN>(g, F2, i, j, k);
  const R e3 = fz<R, false, IN>(g, F3, i, j, k + 1), w3 = fz<R, false, IN>(g, F3, i, j, k);
  // d cp/d mx, d cn/d mn, d/d x, and d/dD = -c/D.  cp = num/Dp: lnum =
  // lcp*h/Dp, lDp = -lnum*(mx-x)/Dp, with one reciprocal per denominator.
  const R lcp = A.lcp.ld(i, j, k), lcn = A.lcn.ld(i, j, k);
  R lnum_p = R(0), lnum_n = R(0), lDp = R(0), lDn = R(0);
  if (nonzero(lcp) || nonzero(lcn)) {
    const R xc = P.xant.ld(i, j, k), hc = P.h.ld(i, j, k);
    const R ep = Eps<R>::v;
    const R Dp = pn(e1) + pp(w1) + pn(e2) + pp(w2) + pn(e3) + pp(w3) + ep;
    const R Dn = pp(e1) + pn(w1) + pp(e2) + pn(w2) + pp(e3) + pn(w3) + ep;
    const R rp = quot(R(1), Dp), rn = quot(R(1), Dn);
    lnum_p = lcp * hc * rp;
    lnum_n = lcn * hc * rn;
    lDp = -(lnum_p * (x.ma.v - xc)) * rp;
    lDn = -(lnum_n * (xc - x.mi.v)) * rn;
  }
  // the adjoint of this pass's extrema: the ratios' part and what the next
  // pass carried back (lmx, lmn)
  const R lma = A.lmx.p ? lnum_p + A.lmx.ld(i, j, k) : lnum_p;
  const R lmi = A.lmn.p ? -lnum_n + A.lmn.ld(i, j, k) : -lnum_n;
  if (!FIRST && x.ma.id == 14) addat(A.lmxp, i, j, k, lma);
  else x.add(A, x.ma.id, i, j, k, lma);
  if (!FIRST && x.mi.id == 14) addat(A.lmnp, i, j, k, lmi);
  else x.add(A, x.mi.id, i, j, k, lmi);
  addat(A.lxant, i, j, k, lnum_n - lnum_p);
  // Dp = pn(e)+pp(w)+..., Dn = pp(e)+pn(w)+... over the six faces
  fx_add<R, false, IN>(g, LF1, i + 1, j, k, lflux(e1, lDp, lDn, false));
  fx_add<R, false, IN>(g, LF1, i, j, k, lflux(w1, lDp, lDn, true));
  fy_add<R, false, IN>(g, LF2, i, j + 1, k, lflux(e2, lDp, lDn, false));
  fy_add<R, false, IN>(g, LF2, i, j, k, lflux(w2, lDp, lDn, true));
  fz_add<R, false, IN>(g, LF3, i, j, k + 1, lflux(e3, lDp, lDn, false));
  fz_add<R, false, IN>(g, LF3, i, j, k, lflux(w3, lDp, lDn, true));
}
// Only a cell whose ratios limit a flux, or whose extrema carry an adjoint
// back, contributes; the rest (about nine in ten on a random field) need no
// fold of 14 values and no quotient.  A warp's row holds a few such cells, so
// the block of 128 packs its cells first and its leading warps take them.
// 256x256x64 FP64: 190 us, 338 with every cell in its own lane; FP32
// 128x128x64: 25 us, 37 before.
template <class R, bool FIRST, bool STD>
__global__ void KA_LB_BOUNDS ka_bounds(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  __shared__ int list[128];
  __shared__ int count;
  const Geo& g = P.g;
  const int k = blockIdx.z + 1;
  const int t = threadIdx.y * 32 + threadIdx.x;
  int i = blockIdx.x * 32 + threadIdx.x + 1, j = blockIdx.y * 4 + threadIdx.y + 1;
  if (t == 0) count = 0;
  __syncthreads();
  bool act = false;
  if (i <= g.np && j <= g.mp) {
    act = nonzero(A.lcp.ld(i, j, k)) || nonzero(A.lcn.ld(i, j, k));
    if (A.lmx.p) act = act || nonzero(A.lmx.ld(i, j, k)) || nonzero(A.lmn.ld(i, j, k));
  }
  const unsigned m = __ballot_sync(0xffffffffu, act);
  int base = 0;
  if (threadIdx.x == 0 && m) base = atomicAdd(&count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (act) list[base + __popc(m & ((1u << threadIdx.x) - 1u))] = t;
  __syncthreads();
  if (t >= count) return;
  const int c = list[t];
  i = blockIdx.x * 32 + (c & 31) + 1;
  j = blockIdx.y * 4 + (c >> 5) + 1;
  if (i >= 2 && i < g.np && j >= 2 && j < g.mp && k >= 2 && k < g.lp) ka_bounds_cell<R, FIRST, STD, true>(P, A, i, j, k);
  else ka_bounds_cell<R, FIRST, STD, false>(P, A, i, j, k);
}

// ---- pseudo-velocity (gauge): v = vdyf(xl,xr,a,hm) - 0.125*a*hm*cr ------------
// cr = S2*rat4(y0,y1,y2,y3) [+ S3*rat4(z0,z1,z2,z3)], S = sums of four a faces.
// AIN: a = the caller's Courant numbers (gradient into gu); otherwise a = the
// previous pass's limited velocities, read with the wall rule (gradient into
// that pass's lambda_w).

// The adjoint of one face's v = K*(xr-xl) - 0.03125*a*hm*cr4, with
// K = (|a| - a*a*hm)/2 and cr4 = S*D [+ S'*D'], the 4-face sums S times the
// unscaled rat4 differences D (4*cr of the forward's form).  U: hm == 1.
template <class R, bool U>
struct FaceAdj {
  R la, lK, lcr4;
  __device__ __forceinline__ FaceAdj(R lv, R a, R hm, R xl, R xrr, R cr4) {
    // the products by powers of two run on the integer pipe (scale_down/up)
    const R K = scale_down<1>(fabs(a) - hmul<U>(a * a, hm));
    la = lv * (scale_down<1>((dabs(a) - hmul<U>(scale_up<1>(a), hm)) * (xrr - xl)) -
               hmul<U>(scale_down<5>(cr4), hm));
    lK = lv * K;
    lcr4 = negv(lv * hmul<U>(scale_down<5>(a), hm));
  }
};

// U: the warp's face densities are all exactly 1.  PS: the pair sums of the
// pass's input field are in cp/cn/q (kf_pairs), as in the forward stage.
// PV (with PS): the velocities' cell-centred pairs are in f1..f3.  Without IN
// (a full warp at a boundary) the stored pairs are read through the boundary
// maps of the values they sum, as in pseudo_form.
template <class R, bool AIN, bool IN, bool U = false, bool PS = false, bool PV = false>
__device__ __forceinline__ void ka_pseudo_cell(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
  const Geo& g = P.g;
  const Arr<R>& X = P.xant;
  const Arr<R>& U1 = AIN ? P.u1 : P.w1;
  const Arr<R>& U2 = AIN ? P.u2 : P.w2;
  const Arr<R>& U3 = AIN ? P.u3 : P.w3;
  const bool zt = IN || g.bz || (k > 1 && k < g.lp);
#define XX(a, b, c) xr<R, IN>(g, X, (a), (b), (c))
#define LX(a, b, c, v) xr_add<R, IN>(g, A.lxant, (a), (b), (c), (v))
#define AX(f, b, c) fx<R, AIN, IN>(g, U1, (f), (b), (c))
#define AY(a, f, c) fy<R, AIN, IN>(g, U2, (a), (f), (c))
#define AZ(a, b, f) fz<R, AIN, IN>(g, U3, (a), (b), (f))
#define MX(a) cx<IN>(g, (a))
#define MY(a) cy<IN>(g, (a))
#define MZ(a) cz<IN>(g, (a))
#define QX(a) xmx<IN>(g, (a))
#define QY(a) xmy<IN>(g, (a))
#define S2X_ (PV ? P.f2.ld(MX(i - 1), j, k) + P.f2.ld(i, j, k) : VSUM_2X)
#define S3X_ (PV ? P.f3.ld(MX(i - 1), j, k) + P.f3.ld(i, j, k) : VSUM_3X)
#define S1Y_ (PV ? P.f1.ld(i, MY(j - 1), k) + P.f1.ld(i, j, k) : VSUM_1Y)
#define S3Y_ (PV ? P.f3.ld(i, MY(j - 1), k) + P.f3.ld(i, j, k) : VSUM_3Y)
#define S1Z_ (PV ? P.f1.ld(i, j, MZ(k - 1)) + P.f1.ld(i, j, k) : VSUM_1Z)
#define S2Z_ (PV ? P.f2.ld(i, j, MZ(k - 1)) + P.f2.ld(i, j, k) : VSUM_2Z)
  // x faces
  if (IN || g.bx || i > 1) {
    const R lv = A.lv1.ld(i, j, k);
    const R hm = U ? R(1) : P.hmx.ld(i, j, k), a = fx<R, AIN, IN>(g, U1, i, j, k);
    const R xl = XX(i - 1, j, k), xrr = XX(i, j, k);
    const R S2 = S2X_;
    const R D2 = PS ? P.cp.ld(i, QY(j + 1), k) - P.cp.ld(i, QY(j - 1), k)
                    : dif4(XX(i - 1, j - 1, k), XX(i, j - 1, k), XX(i - 1, j + 1, k), XX(i, j + 1, k));
    R cr4 = S2 * D2, S3 = R(0), D3 = R(0);
    if (zt) {
      S3 = S3X_;
      D3 = PS ? P.cp.ld(i, j, MZ(k + 1)) - P.cp.ld(i, j, MZ(k - 1))
              : dif4(XX(i - 1, j, k - 1), XX(i, j, k - 1), XX(i - 1, j, k + 1), XX(i, j, k + 1));
      cr4 = cr4 + S3 * D3;
    }
    const FaceAdj<R, U> f(lv, a, hm, xl, xrr, cr4);
    fx_add<R, AIN, IN>(g, A.la1, i, j, k, f.la);
    LX(i, j, k, f.lK);
    LX(i - 1, j, k, negv(f.lK));
    const R lS2 = f.lcr4 * D2, lR2 = f.lcr4 * S2, nR2 = negv(lR2);
    fy_add<R, AIN, IN>(g, A.la2, i - 1, j, k, lS2);
    fy_add<R, AIN, IN>(g, A.la2, i - 1, j + 1, k, lS2);
    fy_add<R, AIN, IN>(g, A.la2, i, j + 1, k, lS2);
    fy_add<R, AIN, IN>(g, A.la2, i, j, k, lS2);
    LX(i, j + 1, k, lR2); LX(i - 1, j + 1, k, lR2); LX(i, j - 1, k, nR2); LX(i - 1, j - 1, k, nR2);
    if (zt) {
      const R lS3 = f.lcr4 * D3, lR3 = f.lcr4 * S3, nR3 = negv(lR3);
      fz_add<R, AIN, IN>(g, A.la3, i - 1, j, k, lS3);
      fz_add<R, AIN, IN>(g, A.la3, i - 1, j, k + 1, lS3);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k + 1, lS3);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k, lS3);
      LX(i, j, k + 1, lR3); LX(i - 1, j, k + 1, lR3); LX(i, j, k - 1, nR3); LX(i - 1, j, k - 1, nR3);
    }
  }
  // y faces
  if (IN || g.by || j > 1) {
    const R lv = A.lv2.ld(i, j, k);
    const R hm = U ? R(1) : P.hmy.ld(i, j, k), a = fy<R, AIN, IN>(g, U2, i, j, k);
    const R xl = XX(i, j - 1, k), xrr = XX(i, j, k);
    const R S1 = S1Y_;
    const R D1 = PS ? P.cn.ld(QX(i + 1), j, k) - P.cn.ld(QX(i - 1), j, k)
                    : dif4(XX(i - 1, j - 1, k), XX(i - 1, j, k), XX(i + 1, j - 1, k), XX(i + 1, j, k));
    R cr4 = S1 * D1, S3 = R(0), D3 = R(0);
    if (zt) {
      S3 = S3Y_;
      D3 = PS ? P.cn.ld(i, j, MZ(k + 1)) - P.cn.ld(i, j, MZ(k - 1))
              : dif4(XX(i, j - 1, k - 1), XX(i, j, k - 1), XX(i, j - 1, k + 1), XX(i, j, k + 1));
      cr4 = cr4 + S3 * D3;
    }
    const FaceAdj<R, U> f(lv, a, hm, xl, xrr, cr4);
    fy_add<R, AIN, IN>(g, A.la2, i, j, k, f.la);
    LX(i, j, k, f.lK);
    LX(i, j - 1, k, negv(f.lK));
    const R lS1 = f.lcr4 * D1, lR1 = f.lcr4 * S1, nR1 = negv(lR1);
    fx_add<R, AIN, IN>(g, A.la1, i, j - 1, k, lS1);
    fx_add<R, AIN, IN>(g, A.la1, i, j, k, lS1);
    fx_add<R, AIN, IN>(g, A.la1, i + 1, j, k, lS1);
    fx_add<R, AIN, IN>(g, A.la1, i + 1, j - 1, k, lS1);
    LX(i + 1, j, k, lR1); LX(i + 1, j - 1, k, lR1); LX(i - 1, j, k, nR1); LX(i - 1, j - 1, k, nR1);
    if (zt) {
      const R lS3 = f.lcr4 * D3, lR3 = f.lcr4 * S3, nR3 = negv(lR3);
      fz_add<R, AIN, IN>(g, A.la3, i, j - 1, k, lS3);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k, lS3);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k + 1, lS3);
      fz_add<R, AIN, IN>(g, A.la3, i, j - 1, k + 1, lS3);
      LX(i, j, k + 1, lR3); LX(i, j - 1, k + 1, lR3); LX(i, j, k - 1, nR3); LX(i, j - 1, k - 1, nR3);
    }
  }
  // z faces
  if (IN || g.bz || k > 1) {
    const R lv = A.lv3.ld(i, j, k);
    const R hm = U ? R(1) : P.hmz.ld(i, j, k), a = fz<R, AIN, IN>(g, U3, i, j, k);
    const R xl = XX(i, j, k - 1), xrr = XX(i, j, k);
    const R S1 = S1Z_;
    const R D1 = PS ? P.q.ld(QX(i + 1), j, k) - P.q.ld(QX(i - 1), j, k)
                    : dif4(XX(i - 1, j, k - 1), XX(i - 1, j, k), XX(i + 1, j, k - 1), XX(i + 1, j, k));
    const R S2 = S2Z_;
    const R D2 = PS ? P.q.ld(i, QY(j + 1), k) - P.q.ld(i, QY(j - 1), k)
                    : dif4(XX(i, j - 1, k - 1), XX(i, j - 1, k), XX(i, j + 1, k - 1), XX(i, j + 1, k));
    const R cr4 = S1 * D1 + S2 * D2;
    const FaceAdj<R, U> f(lv, a, hm, xl, xrr, cr4);
    fz_add<R, AIN, IN>(g, A.la3, i, j, k, f.la);
    LX(i, j, k, f.lK);
    LX(i, j, k - 1, negv(f.lK));
    const R lS1 = f.lcr4 * D1, lR1 = f.lcr4 * S1, nR1 = negv(lR1);
    fx_add<R, AIN, IN>(g, A.la1, i, j, k - 1, lS1);
    fx_add<R, AIN, IN>(g, A.la1, i, j, k, lS1);
    fx_add<R, AIN, IN>(g, A.la1, i + 1, j, k, lS1);
    fx_add<R, AIN, IN>(g, A.la1, i + 1, j, k - 1, lS1);
    LX(i + 1, j, k, lR1); LX(i + 1, j, k - 1, lR1); LX(i - 1, j, k, nR1); LX(i - 1, j, k - 1, nR1);
    const R lS2 = f.lcr4 * D2, lR2 = f.lcr4 * S2, nR2 = negv(lR2);
    fy_add<R, AIN, IN>(g, A.la2, i, j, k - 1, lS2);
    fy_add<R, AIN, IN>(g, A.la2, i, j + 1, k - 1, lS2);
    fy_add<R, AIN, IN>(g, A.la2, i, j + 1, k, lS2);
    fy_add<R, AIN, IN>(g, A.la2, i, j, k, lS2);
    LX(i, j + 1, k, lR2); LX(i, j + 1, k - 1, lR2); LX(i, j - 1, k, nR2); LX(i, j - 1, k - 1, nR2);
  }
#undef XX
#undef LX
#undef AX
#undef AY
#undef AZ
#undef MX
#undef MY
#undef MZ
#undef QX
#undef QY
#undef S2X_
#undef S3X_
#undef S1Y_
#undef S3Y_
#undef S1Z_
#undef S2Z_
}
template <class R, bool AIN>
__global__ void KA_LB_PSEUDO ka_pseudo(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  const bool win = warp_interior(P.g, i, j, k);
  // every pair sum is stored: full warps at a boundary read them too
  const bool pin = !win && warp_on_grid(P.g, i, j);
  if (i > P.g.np || j > P.g.mp) return;
  if (pin) {
    if (warp_unit_faces(P, i, j, k))
      ka_pseudo_cell<R, AIN, false, true, true, true>(P, A, i, j, k);
    else
      ka_pseudo_cell<R, AIN, false, false, true, true>(P, A, i, j, k);
  } else if (!win) {
    ka_pseudo_cell<R, AIN, false>(P, A, i, j, k);
  } else if (warp_unit_faces(P, i, j, k)) {  // FP64
    ka_pseudo_cell<R, AIN, true, true, true, true>(P, A, i, j, k);
  } else {
    ka_pseudo_cell<R, AIN, true, false, true, true>(P, A, i, j, k);
  }
}

// The same reverse in gather form (FP32, every axis periodic): the scatter
// above adds 57 values a cell by atomics, and at four bytes each the L2's
// atomic rate bounds it.  The additions of a face go to cells and faces that
// differ by a shift, so their sums over the two faces of a cell on each axis
// are six cell-centred fields:
//   T1 (T2, T3): R of the faces whose cross difference runs along x (y, z);
//                lambda_x(i) gains T1(i-1) - T1(i+1), and so on
//   C1 (C2, C3): the products on the 4-face sums of u1 (u2, u3);
//                lambda_a1 of face i gains C1(i-1) + C1(i), and so on
// A first kernel forms them (each face twice, once from either cell: FP64,
// bound by its pipe, keeps the scatter) with what goes to the cell and its
// lower faces themselves, a second one adds the shifted sums.  The pair sums
// and velocity pairs come from kf_pairs, the six fields from the standard
// form's accumulators.
// Both kernels are bound by issue and load latency: the workspace's fields have
// one layout, so a cell is one offset in all of them and a neighbour one
// difference, instead of index arithmetic per load (850 instructions a cell
// before).  128x128x64: 28 + 13 us (44 + 14 with it), 89 by scatter.
template <class R, bool AIN>
__global__ void __launch_bounds__(128) ka_cross(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  ACELL
  const Nbr<R> n(g, P.cp, i, j, k);
  const long o = n.o;
  const Arr<R>& U1 = AIN ? P.u1 : P.w1;
  const Arr<R>& U2 = AIN ? P.u2 : P.w2;
  const Arr<R>& U3 = AIN ? P.u3 : P.w3;
  const R* const u1 = U1.p + U1.off(i, j, k);
  const R* const u2 = U2.p + U2.off(i, j, k);
  const R* const u3 = U3.p + U3.off(i, j, k);
  const R* const X = P.xant.p + P.xant.off(i, j, k);
  const R *const cp = P.cp.p + o, *const cn = P.cn.p + o, *const q = P.q.p + o;
  const R *const F1 = P.f1.p + o, *const F2 = P.f2.p + o, *const F3 = P.f3.p + o;
  const R *const lv1 = A.lv1.p + o, *const lv2 = A.lv2.p + o, *const lv3 = A.lv3.p + o;
  const R *const hx = P.hmx.p + o, *const hy = P.hmy.p + o, *const hz = P.hmz.p + o;
  const R x = X[0], f1 = F1[0], f2 = F2[0], f3 = F3[0];
  R lx, C1, C2, C3, T1, T2, T3, la1, la2, la3;
  {  // x: cross differences along y and z; the lower face, then the upper one
    const R S2 = F2[n.xm] + f2, S3 = F3[n.xm] + f3, D2 = cp[n.yp] - cp[n.ym], D3 = cp[n.zp] - cp[n.zm];
    const FaceAdj<R, false> f(lv1[0], u1[0], hx[0], X[n.xm], x, S2 * D2 + S3 * D3);
    la1 = f.la;
    C2 = f.lcr4 * D2;
    T2 = f.lcr4 * S2;
    C3 = f.lcr4 * D3;
    T3 = f.lcr4 * S3;
    lx = f.lK;
  }
  {
    const R S2 = f2 + F2[n.xp], S3 = f3 + F3[n.xp], D2 = cp[n.xp + n.yp] - cp[n.xp + n.ym],
            D3 = cp[n.xp + n.zp] - cp[n.xp + n.zm];
    const FaceAdj<R, false> f(lv1[n.xp], u1[n.xp], hx[n.xp], x, x, R(0));
    C2 += f.lcr4 * D2;
    T2 += f.lcr4 * S2;
    C3 += f.lcr4 * D3;
    T3 += f.lcr4 * S3;
    lx -= f.lK;
  }
  {  // y: along x and z
    const int ux = (j < g.mp ? 1 : 1 - g.mp) * U2.sy;
    const R S1 = F1[n.ym] + f1, S3 = F3[n.ym] + f3, D1 = cn[n.xp] - cn[n.xm], D3 = cn[n.zp] - cn[n.zm];
    const FaceAdj<R, false> f(lv2[0], u2[0], hy[0], X[(j > 1 ? -1 : g.mp - 1) * P.xant.sy], x, S1 * D1 + S3 * D3);
    la2 = f.la;
    C1 = f.lcr4 * D1;
    T1 = f.lcr4 * S1;
    C3 += f.lcr4 * D3;
    T3 += f.lcr4 * S3;
    lx += f.lK;
    const R S1p = f1 + F1[n.yp], S3p = f3 + F3[n.yp], D1p = cn[n.yp + n.xp] - cn[n.yp + n.xm],
            D3p = cn[n.yp + n.zp] - cn[n.yp + n.zm];
    const FaceAdj<R, false> p(lv2[n.yp], u2[ux], hy[n.yp], x, x, R(0));
    C1 += p.lcr4 * D1p;
    T1 += p.lcr4 * S1p;
    C3 += p.lcr4 * D3p;
    T3 += p.lcr4 * S3p;
    lx -= p.lK;
  }
  {  // z: along x and y
    const long ux = (long)(k < g.lp ? 1 : 1 - g.lp) * U3.sz, xz = (long)(k > 1 ? -1 : g.lp - 1) * P.xant.sz;
    const R S1 = F1[n.zm] + f1, S2 = F2[n.zm] + f2, D1 = q[n.xp] - q[n.xm], D2 = q[n.yp] - q[n.ym];
    const FaceAdj<R, false> f(lv3[0], u3[0], hz[0], X[xz], x, S1 * D1 + S2 * D2);
    la3 = f.la;
    C1 += f.lcr4 * D1;
    T1 += f.lcr4 * S1;
    C2 += f.lcr4 * D2;
    T2 += f.lcr4 * S2;
    lx += f.lK;
    const R S1p = f1 + F1[n.zp], S2p = f2 + F2[n.zp], D1p = q[n.zp + n.xp] - q[n.zp + n.xm],
            D2p = q[n.zp + n.yp] - q[n.zp + n.ym];
    const FaceAdj<R, false> p(lv3[n.zp], u3[ux], hz[n.zp], x, x, R(0));
    C1 += p.lcr4 * D1p;
    T1 += p.lcr4 * S1p;
    C2 += p.lcr4 * D2p;
    T2 += p.lcr4 * S2p;
    lx -= p.lK;
  }
  A.lxant.p[o] += lx;
  addat(A.la1, i, j, k, la1);  // the caller's gradients: steps on other streams may add to them
  addat(A.la2, i, j, k, la2);
  addat(A.la3, i, j, k, la3);
  A.lg1.p[o] = C1;
  A.lg2.p[o] = C2;
  A.lg3.p[o] = C3;
  A.lf1.p[o] = T1;
  A.lf2.p[o] = T2;
  A.lf3.p[o] = T3;
}
template <class R>
__global__ void __launch_bounds__(128) ka_cross_sum(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  ACELL
  const Nbr<R> n(g, A.lg1, i, j, k);
  const long o = n.o;
  const R *const g1 = A.lg1.p + o, *const g2 = A.lg2.p + o, *const g3 = A.lg3.p + o;
  const R *const t1 = A.lf1.p + o, *const t2 = A.lf2.p + o, *const t3 = A.lf3.p + o;
  const R lx = A.lxant.p[o] + ((t1[n.xm] - t1[n.xp]) + (t2[n.ym] - t2[n.yp]) + (t3[n.zm] - t3[n.zp]));
  A.lxant.p[o] = lx;
  addat(A.la1, i, j, k, g1[n.xm] + g1[0]);
  addat(A.la2, i, j, k, g2[n.ym] + g2[0]);
  addat(A.la3, i, j, k, g3[n.zm] + g3[0]);
}

// ---- standard form (antidiff3d-standard-gpubc.f90) ---------------------------
// update: x_out = rhr*(q - d*hinv), d = signed sum of the limited fluxes g
template <class R, bool IN>
__device__ __forceinline__ void ka_update_std_cell(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
  const Geo& g = P.g;
  const R lt = P.rhr.ld(i, j, k) * A.lam.ld(i, j, k);
  if (A.lx.p) A.lx.at(i, j, k) = R(0);  // as the gauge form's update
  addat(A.lq, i, j, k, lt);
  const R lD = -lt * P.hinv.ld(i, j, k);
  fx_add<R, false, IN>(g, A.lg1, i + 1, j, k, lD);
  fx_add<R, false, IN>(g, A.lg1, i, j, k, -lD);
  fy_add<R, false, IN>(g, A.lg2, i, j + 1, k, lD);
  fy_add<R, false, IN>(g, A.lg2, i, j, k, -lD);
  fz_add<R, false, IN>(g, A.lg3, i, j, k + 1, lD);
  fz_add<R, false, IN>(g, A.lg3, i, j, k, -lD);
}
template <class R>
__global__ void __launch_bounds__(128) ka_update_std(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
#define C(IN) ka_update_std_cell<R, IN>(P, A, i, j, k)
  ADISPATCH(C)
#undef C
}

// limiter: w = vlim_std(v, a1, a2, x(c-1), x(c)) with a1 = min3(cp(c), cn(c-1)),
// a2 = min3(cp(c-1), cn(c)); g = donor(q(c-1), q(c), w).  possign() is
// piecewise constant: only v, a1 and a2 carry a derivative through it.
template <class R, bool NONOS, bool IN>
__device__ __forceinline__ void ka_limit_std_cell(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
  const Geo& g = P.g;
  const Arr<R>& X = P.xant;
  const R cpc = NONOS ? P.cp.ld(i, j, k) : R(0), cnc = NONOS ? P.cn.ld(i, j, k) : R(0);
  const R xc = X.ld(i, j, k), qc = P.q.ld(i, j, k);
#define LIMIT_STD_FACE(V, LV, LW, LG, IM, JM, KM)                                                       \
  {                                                                                                     \
    const R v = V.ld(i, j, k);                                                                          \
    const R xl = X.ld(IM, JM, KM), ql = P.q.ld(IM, JM, KM);                                             \
    R w = v, a1 = R(0), a2 = R(0), cpm = R(0), cnm = R(0);                                              \
    if (NONOS) {                                                                                        \
      cpm = P.cp.ld(IM, JM, KM);                                                                        \
      cnm = P.cn.ld(IM, JM, KM);                                                                        \
      a1 = min3(cpc, cnm);                                                                              \
      a2 = min3(cpm, cnc);                                                                              \
      w = vlim_std(v, a1, a2, xl, xc);                                                                  \
    }                                                                                                   \
    const R lg = LG.ld(i, j, k);                                                                        \
    addat(A.lq, IM, JM, KM, lg * pp(w));                                                                \
    addat(A.lq, i, j, k, -lg * pn(w));                                                                  \
    const R lw = LW.ld(i, j, k) + lg * (dpp(w) * ql - dpn(w) * qc);                                     \
    if (!NONOS) {                                                                                       \
      addat(LV, i, j, k, lw);                                                                           \
    } else {                                                                                            \
      const R sl = possign(xl), sml = possign(-xl), sr = possign(xc), smr = possign(-xc);              \
      addat(LV, i, j, k, lw * (dpp(v) * (a1 * sl + a2 * sml) - dpn(v) * (a2 * sr + a1 * smr)));         \
      min3_adj(cpc, cnm, lw * (pp(v) * sl - pn(v) * smr), A.lcp, i, j, k, A.lcn, IM, JM, KM);          \
      min3_adj(cpm, cnc, lw * (pp(v) * sml - pn(v) * sr), A.lcp, IM, JM, KM, A.lcn, i, j, k);          \
    }                                                                                                   \
  }
  if (IN || g.bx || i > 1) LIMIT_STD_FACE(P.v1, A.lv1, A.lw1, A.lg1, (IN ? i - 1 : wrapi(i - 1, g.np)), j, k)
  if (IN || g.by || j > 1) LIMIT_STD_FACE(P.v2, A.lv2, A.lw2, A.lg2, i, (IN ? j - 1 : wrapi(j - 1, g.mp)), k)
  if (IN || g.bz || k > 1) LIMIT_STD_FACE(P.v3, A.lv3, A.lw3, A.lg3, i, j, (IN ? k - 1 : wrapi(k - 1, g.lp)))
#undef LIMIT_STD_FACE
}
template <class R, bool NONOS>
__global__ void __launch_bounds__(128) ka_limit_std(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
#define C(IN) ka_limit_std_cell<R, NONOS, IN>(P, A, i, j, k)
  ADISPATCH(C)
#undef C
}

// vcorra(a, b, y1, y2, hm) = -(0.125*a*b*y1*hm/y2) with y1 = (|p1|+|p2|)-(|m1|+|m2|),
// y2 = |p1|+|p2|+|m1|+|m2|+ep; returns dv/da and dv/db, scatters dv/dx.
template <class R>
struct VcTerm {
  R lb;  // lambda of b
  R la;  // lambda of a
};
template <class R, bool IN>
__device__ __forceinline__ VcTerm<R> vcorra_adj(const Geo& g, const Arr<R>& X, const Arr<R>& LX, R lv, R a, R b,
                                                R hm, int pi1, int pj1, int pk1, int pi2, int pj2, int pk2,
                                                int mi1, int mj1, int mk1, int mi2, int mj2, int mk2) {
  const R p1 = xr<R, IN>(g, X, pi1, pj1, pk1), p2 = xr<R, IN>(g, X, pi2, pj2, pk2);
  const R m1 = xr<R, IN>(g, X, mi1, mj1, mk1), m2 = xr<R, IN>(g, X, mi2, mj2, mk2);
  const R y1 = (fabs(p1) + fabs(p2)) - (fabs(m1) + fabs(m2));
  const R y2 = fabs(p1) + fabs(p2) + fabs(m1) + fabs(m2) + Eps<R>::v;
  const R t = -R(0.125) * hm;
  const R dy1 = quot(t * a * b, y2), dy2 = quot(-t * a * b * y1, y2 * y2);
  xr_add<R, IN>(g, LX, pi1, pj1, pk1, lv * (dy1 + dy2) * dabs(p1));
  xr_add<R, IN>(g, LX, pi2, pj2, pk2, lv * (dy1 + dy2) * dabs(p2));
  xr_add<R, IN>(g, LX, mi1, mj1, mk1, lv * (dy2 - dy1) * dabs(m1));
  xr_add<R, IN>(g, LX, mi2, mj2, mk2, lv * (dy2 - dy1) * dabs(m2));
  return VcTerm<R>{quot(lv * t * a * y1, y2), quot(lv * t * b * y1, y2)};
}

// pseudo-velocity: f*ns = donor(xl, xr, v) first, then
// v = vdyfa(xl, xr, a, hm) + vcorra(cross 1) [+ vcorra(cross 2)], and the
// q = x/rhr of the limiter's fluxes back into x.
template <class R, bool AIN, bool IN>
__device__ __forceinline__ void ka_pseudo_std_cell(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
  const Geo& g = P.g;
  const Arr<R>& X = P.xant;
  const Arr<R>& U1 = AIN ? P.u1 : P.w1;
  const Arr<R>& U2 = AIN ? P.u2 : P.w2;
  const Arr<R>& U3 = AIN ? P.u3 : P.w3;
  const R ep = Eps<R>::v;
  const bool zt = IN || g.bz || (k > 1 && k < g.lp);
  addat(A.lxant, i, j, k, quot(A.lq.ld(i, j, k), P.rhr.ld(i, j, k)));
#define XX(a, b, c) xr<R, IN>(g, X, (a), (b), (c))
#define LX(a, b, c, v) xr_add<R, IN>(g, A.lxant, (a), (b), (c), (v))
#define AX(f, b, c) fx<R, AIN, IN>(g, U1, (f), (b), (c))
#define AY(a, f, c) fy<R, AIN, IN>(g, U2, (a), (f), (c))
#define AZ(a, b, f) fz<R, AIN, IN>(g, U3, (a), (b), (f))
  // the face's own velocity, donor flux and vdyfa; returns lambda of v after f*ns
#define FACE_HEAD(LV, LF, V, AF, HM, XLI, XLJ, XLK)                                                     \
  const R v = V.ld(i, j, k), hm = HM.ld(i, j, k), a = AF;                                           \
  const R xl = XX(XLI, XLJ, XLK), xrr = XX(i, j, k);                                                \
  const R lf = LF.ld(i, j, k);                                                                      \
  LX(XLI, XLJ, XLK, lf * pp(v));                                                                    \
  LX(i, j, k, -lf * pn(v));                                                                         \
  const R lv = LV.ld(i, j, k) + lf * (dpp(v) * xl - dpn(v) * xrr);                                  \
  const R K = fabs(a) - a * a * hm, N = fabs(xrr) - fabs(xl), Dd = fabs(xrr) + fabs(xl) + ep;       \
  R la = quot(lv * (dabs(a) - R(2) * a * hm) * N, Dd);                                              \
  LX(i, j, k, quot(lv * K * dabs(xrr) * (Dd - N), Dd * Dd));                                        \
  LX(XLI, XLJ, XLK, quot(-lv * K * dabs(xl) * (Dd + N), Dd * Dd));
  if (IN || g.bx || i > 1) {
    FACE_HEAD(A.lv1, A.lf1, P.v1, (fx<R, AIN, IN>(g, U1, i, j, k)), P.hmx, i - 1, j, k)
    {
      const R b = VSUM_2X;
      const VcTerm<R> c = vcorra_adj<R, IN>(g, X, A.lxant, lv, a, b, hm, i - 1, j + 1, k, i, j + 1, k, i - 1, j - 1, k,
                                        i, j - 1, k);
      la += c.la;
      fy_add<R, AIN, IN>(g, A.la2, i - 1, j, k, c.lb);
      fy_add<R, AIN, IN>(g, A.la2, i - 1, j + 1, k, c.lb);
      fy_add<R, AIN, IN>(g, A.la2, i, j + 1, k, c.lb);
      fy_add<R, AIN, IN>(g, A.la2, i, j, k, c.lb);
    }
    if (zt) {
      const R b = VSUM_3X;
      const VcTerm<R> c = vcorra_adj<R, IN>(g, X, A.lxant, lv, a, b, hm, i - 1, j, k + 1, i, j, k + 1, i - 1, j, k - 1,
                                        i, j, k - 1);
      la += c.la;
      fz_add<R, AIN, IN>(g, A.la3, i - 1, j, k, c.lb);
      fz_add<R, AIN, IN>(g, A.la3, i - 1, j, k + 1, c.lb);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k + 1, c.lb);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k, c.lb);
    }
    fx_add<R, AIN, IN>(g, A.la1, i, j, k, la);
  }
  if (IN || g.by || j > 1) {
    FACE_HEAD(A.lv2, A.lf2, P.v2, (fy<R, AIN, IN>(g, U2, i, j, k)), P.hmy, i, j - 1, k)
    {
      const R b = VSUM_1Y;
      const VcTerm<R> c = vcorra_adj<R, IN>(g, X, A.lxant, lv, a, b, hm, i + 1, j - 1, k, i + 1, j, k, i - 1, j - 1, k,
                                        i - 1, j, k);
      la += c.la;
      fx_add<R, AIN, IN>(g, A.la1, i, j - 1, k, c.lb);
      fx_add<R, AIN, IN>(g, A.la1, i, j, k, c.lb);
      fx_add<R, AIN, IN>(g, A.la1, i + 1, j, k, c.lb);
      fx_add<R, AIN, IN>(g, A.la1, i + 1, j - 1, k, c.lb);
    }
    if (zt) {
      const R b = VSUM_3Y;
      const VcTerm<R> c = vcorra_adj<R, IN>(g, X, A.lxant, lv, a, b, hm, i, j - 1, k + 1, i, j, k + 1, i, j - 1, k - 1,
                                        i, j, k - 1);
      la += c.la;
      fz_add<R, AIN, IN>(g, A.la3, i, j - 1, k, c.lb);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k, c.lb);
      fz_add<R, AIN, IN>(g, A.la3, i, j, k + 1, c.lb);
      fz_add<R, AIN, IN>(g, A.la3, i, j - 1, k + 1, c.lb);
    }
    fy_add<R, AIN, IN>(g, A.la2, i, j, k, la);
  }
  if (IN || g.bz || k > 1) {
    FACE_HEAD(A.lv3, A.lf3, P.v3, (fz<R, AIN, IN>(g, U3, i, j, k)), P.hmz, i, j, k - 1)
    {
      const R b = VSUM_1Z;
      const VcTerm<R> c = vcorra_adj<R, IN>(g, X, A.lxant, lv, a, b, hm, i + 1, j, k - 1, i + 1, j, k, i - 1, j, k - 1,
                                        i - 1, j, k);
      la += c.la;
      fx_add<R, AIN, IN>(g, A.la1, i, j, k - 1, c.lb);
      fx_add<R, AIN, IN>(g, A.la1, i, j, k, c.lb);
      fx_add<R, AIN, IN>(g, A.la1, i + 1, j, k, c.lb);
      fx_add<R, AIN, IN>(g, A.la1, i + 1, j, k - 1, c.lb);
    }
    {
      const R b = VSUM_2Z;
      const VcTerm<R> c = vcorra_adj<R, IN>(g, X, A.lxant, lv, a, b, hm, i, j + 1, k - 1, i, j + 1, k, i, j - 1, k - 1,
                                        i, j - 1, k);
      la += c.la;
      fy_add<R, AIN, IN>(g, A.la2, i, j, k - 1, c.lb);
      fy_add<R, AIN, IN>(g, A.la2, i, j + 1, k - 1, c.lb);
      fy_add<R, AIN, IN>(g, A.la2, i, j + 1, k, c.lb);
      fy_add<R, AIN, IN>(g, A.la2, i, j, k, c.lb);
    }
    fz_add<R, AIN, IN>(g, A.la3, i, j, k, la);
  }
#undef FACE_HEAD
#undef XX
#undef LX
#undef AX
#undef AY
#undef AZ
}
template <class R, bool AIN>
__global__ void __launch_bounds__(128) ka_pseudo_std(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
#define C(IN) ka_pseudo_std_cell<R, AIN, IN>(P, A, i, j, k)
  ADISPATCH(C)
#undef C
}

// ---- upwind: xant = rhr*(x - D*hinv), D = signed sum of donor fluxes --------
// F = donor(xl, xr, u) = pp(u)*xl - pn(u)*xr; dF/du = [u>0]*xl + [u<0]*xr.
// Open-wall neighbours come from bcx/bcy (constants: no gradient).
//
// A cell owns its lower face on each axis (the last cell of an open axis the
// upper one as well) and forms that face's lambda_F from both of its cells:
// three fluxes a cell instead of six, one atomic each to the donor cell and to the
// velocity gradient (steps on other streams may add to the same gradients).
// 256x256x64 FP64: 116 us (142 with a plain read and write of the gradients);
// six fluxes from a cell and a copy of the result 167.
// MF (density step): the step also outputs each face's upwind flux as part
// of its mass flux: the lower face's flux of every cell (u1(i), u2(j), u3(k))
// and the upper face's of the last cell along each axis (u1(np+1), ...),
// which a periodic axis takes from face 1.  Their cotangents add to the
// fluxes' own; at a z wall the flux stored for face 1 is -F3(2) and the one
// for face lp+1 is -F3(lp).
template <class R>
__device__ __forceinline__ void flux_adj(R lF, R u, R xl, R xr_, R* GU, const Arr<R>& Lx, bool l_var, int li, int lj,
                                         int lk, bool r_var, int ri, int rj, int rk) {
  const R m = lF * u;
  if (sgn(u)) {
    if (r_var) addat(Lx, ri, rj, rk, m);
  } else {
    if (l_var) addat(Lx, li, lj, lk, m);
  }
  if (nonzero(u)) atomicAdd(GU, lF * (sgn(u) ? xr_ : xl));
}

// U: rhr and hinv are exactly 1 at the cells read (x*1 == x); an instantiation,
// as a test inside the body became selects between products computed anyway.
template <class R, bool IN, bool MF, bool U>
__device__ __forceinline__ void ka_upwind_cell(const Prob<R>& P, const AdjArr<R>& A, int i, int j, int k) {
  const Geo& g = P.g;
  const Arr<R>& psi = P.psi;
  // the adjoint of a cell's divergence
  auto div = [&](int a, int b, int c) {
    const R l = negv(A.lxant.ld(a, b, c));
    return U ? l : l * P.rhr.ld(a, b, c) * P.hinv.ld(a, b, c);
  };
  {
    const R l = A.lxant.ld(i, j, k);
    addat(A.lx, i, j, k, U ? l : l * P.rhr.ld(i, j, k));
  }
  const R lD = div(i, j, k), x = psi.ld(i, j, k);
  const long bx0 = (long)(j - 1) + (long)g.mp * (k - 1), bxs = (long)g.mp * g.lp;
  const long by0 = (long)(i - 1) + (long)g.np * (k - 1), bys = (long)g.np * g.lp;
  {
    const bool var = IN || i > 1 || g.bx;
    const int im = IN ? i - 1 : wrapi(i - 1, g.np);
    R lF = (var ? div(im, j, k) : R(0)) - lD;
    if (MF) {
      lF += A.lm1.ld(i, j, k);
      if (!IN && i == 1 && g.bx) lF += A.lm1.ld(g.np + 1, j, k);
    }
    flux_adj(lF, P.u1.ld(i, j, k), var ? psi.ld(im, j, k) : P.bcx[bx0], x, &A.gu1.at(i, j, k), A.lx, var, im, j, k,
             true, i, j, k);
    if (!IN && i == g.np && !g.bx)
      flux_adj(MF ? lD + A.lm1.ld(i + 1, j, k) : lD, P.u1.ld(i + 1, j, k), x, P.bcx[bx0 + bxs],
               &A.gu1.at(i + 1, j, k), A.lx, true, i, j, k, false, i, j, k);
  }
  {
    const bool var = IN || j > 1 || g.by;
    const int jm = IN ? j - 1 : wrapi(j - 1, g.mp);
    R lF = (var ? div(i, jm, k) : R(0)) - lD;
    if (MF) {
      lF += A.lm2.ld(i, j, k);
      if (!IN && j == 1 && g.by) lF += A.lm2.ld(i, g.mp + 1, k);
    }
    flux_adj(lF, P.u2.ld(i, j, k), var ? psi.ld(i, jm, k) : P.bcy[by0], x, &A.gu2.at(i, j, k), A.lx, var, i, jm, k,
             true, i, j, k);
    if (!IN && j == g.mp && !g.by)
      flux_adj(MF ? lD + A.lm2.ld(i, j + 1, k) : lD, P.u2.ld(i, j + 1, k), x, P.bcy[by0 + bys],
               &A.gu2.at(i, j + 1, k), A.lx, true, i, j, k, false, i, j, k);
  }
  if (IN || g.bz || k > 1) {
    const int km = IN ? k - 1 : wrapi(k - 1, g.lp);
    const bool wall = !g.bz;
    const R dl = div(i, j, km);
    // F3(1) = -F3(2) and F3(lp+1) = -F3(lp): a wall cell reads its inner face twice
    R lF = (wall && k == 2 ? scale_up<1>(dl) : dl) - (wall && k == g.lp ? scale_up<1>(lD) : lD);
    if (MF) {
      lF += A.lm3.ld(i, j, k);
      if (wall && k == 2) lF -= A.lm3.ld(i, j, 1);
      if (!IN && wall && k == g.lp) lF -= A.lm3.ld(i, j, g.lp + 1);
      if (!IN && g.bz && k == 1) lF += A.lm3.ld(i, j, g.lp + 1);
    }
    flux_adj(lF, P.u3.ld(i, j, k), psi.ld(i, j, km), x, &A.gu3.at(i, j, k), A.lx, true, i, j, km, true, i, j, k);
  }
}
template <class R, bool MF = false>
__global__ void KA_LB_UPWIND ka_upwind(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  const bool win = warp_interior(P.g, i, j, k);
  if (i > P.g.np || j > P.g.mp) return;
  if (!win) {
    ka_upwind_cell<R, false, MF, false>(P, A, i, j, k);
    return;
  }
  if constexpr (sizeof(R) == 8) {
    auto one = [&](int a, int b, int c) { return is_one(P.rhr.ld(a, b, c)) && is_one(P.hinv.ld(a, b, c)); };
    if (__all_sync(0xffffffffu, one(i, j, k) && one(i - 1, j, k) && one(i, j - 1, k) && one(i, j, k - 1))) {
      ka_upwind_cell<R, true, MF, true>(P, A, i, j, k);
      return;
    }
  }
  ka_upwind_cell<R, true, MF, false>(P, A, i, j, k);
}

// Density step: the mass flux of every face adds the last pass's limited
// flux as the forward reads it (fx/fy/fz of the stored faces: the periodic
// wrap, the zero open walls, the mirrored z faces), so its cotangent goes to
// that flux's adjoint through the same read maps.
template <class R>
__global__ void __launch_bounds__(128) ka_mass_to_w(const Prob<R> P, const AdjArr<R> A) {
  chain_begin();
  ACELL
  fx_add<R, false>(g, A.lw1, i, j, k, A.lm1.ld(i, j, k));
  fy_add<R, false>(g, A.lw2, i, j, k, A.lm2.ld(i, j, k));
  fz_add<R, false>(g, A.lw3, i, j, k, A.lm3.ld(i, j, k));
  if (i == g.np) fx_add<R, false>(g, A.lw1, g.np + 1, j, k, A.lm1.ld(g.np + 1, j, k));
  if (j == g.mp) fy_add<R, false>(g, A.lw2, i, g.mp + 1, k, A.lm2.ld(i, g.mp + 1, k));
  if (k == g.lp) fz_add<R, false>(g, A.lw3, i, j, g.lp + 1, A.lm3.ld(i, j, g.lp + 1));
}

// Reverse of the density step's outputs (rho_out_body): x_incomp = x*h,
// pexr1 = x_incomp*pexe, pexr2 = x_incomp, rhr = rhoadv/x_incomp with rhoadv
// the x_incomp input.  lam (dJ/dpsi after the step) gains h*dJ/dx_incomp;
// g_xinc and g_pexe receive dJ/d(x_incomp input) and dJ/dpexe.  Null
// cotangent arrays are zeros.
template <class R>
__global__ void __launch_bounds__(128) ka_rho_out(const Prob<R> P, const Arr<R> out, const Arr<R> lxc,
                                                  const Arr<R> lp1, const Arr<R> lp2, const Arr<R> lrh, Arr<R> lam,
                                                  Arr<R> g_xinc, Arr<R> g_pexe) {
  chain_begin();
  ACELL
  (void)g;
  const R h = P.h.ld(i, j, k);
  const R xc = out.ld(i, j, k) * h;
  const R pe = P.pexe.ld(i, j, k), ra = P.x_incomp.ld(i, j, k);
  const R a_xc = lxc.p ? lxc.ld(i, j, k) : R(0), a_p1 = lp1.p ? lp1.ld(i, j, k) : R(0),
          a_p2 = lp2.p ? lp2.ld(i, j, k) : R(0), a_rh = lrh.p ? lrh.ld(i, j, k) : R(0);
  const R l_xc = a_xc + a_p1 * pe + a_p2 - quot(a_rh * quot(ra, xc), xc);
  lam.at(i, j, k) = lam.ld(i, j, k) + l_xc * h;
  g_xinc.at(i, j, k) = quot(a_rh, xc);
  g_pexe.at(i, j, k) = a_p1 * xc;
}

// J's seed: lambda = psi_N - target on the interior, 0 on the halo.
template <class R>
__global__ void __launch_bounds__(128) ka_seed(const Prob<R> P, const Arr<R> psi, const Arr<R> target, Arr<R> lam) {
  chain_begin();
  ACELL
  lam.at(i, j, k) = psi.ld(i, j, k) - target.ld(i, j, k);
}

// forward record kernels (psi's halo is left untouched: HALO=false); warps
// away from every wall take the bodies without boundary maps, as the
// forward stage kernels do
#define FCELL(BODY)                                          \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;  \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;  \
  const int k = blockIdx.z + 1;                              \
  const bool win = warp_interior(P.g, i, j, k);              \
  if (i > P.g.np || j > P.g.mp) return;                      \
  if (win) {                                                 \
    BODY(true);                                              \
  } else {                                                   \
    BODY(false);                                             \
  }
// As FCELL, with the unit-density instantiation BODY(IN, U) for interior
// warps whose densities are all exactly 1 (FP64).
#define FCELL_U(BODY)                                        \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;  \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;  \
  const int k = blockIdx.z + 1;                              \
  const bool win = warp_interior(P.g, i, j, k);              \
  if (i > P.g.np || j > P.g.mp) return;                      \
  if (!win) {                                                \
    BODY(false, false);                                      \
  } else if (warp_unit_cell(P, i, j, k)) {                   \
    BODY(true, true);                                        \
  } else {                                                   \
    BODY(true, false);                                       \
  }
template <class R>
__global__ void __launch_bounds__(128, (KfMinBlocks<R, 8, 10>::v)) kf_upwind(const Prob<R> P) {
  chain_begin();
#define B(IN, U) upwind_body<R, true, false, IN, U>(P, i, j, k)
  FCELL_U(B)
#undef B
}
template <class R, bool AIN, bool PV>
__global__ void __launch_bounds__(128) kf_pairs(const Prob<R> P) {
  chain_begin();
  ACELL
  (void)g;
  pairs_body<R, AIN, PV>(P, i, j, k);
}
// the forward stage's dispatch: unit face densities and pair sums (FP64),
// and the stage kernel's seven resident blocks per SM for FP64
template <class R>
struct KfPseudoMinBlocks {
  static constexpr int v = sizeof(R) == 8 ? 7 : 1;
};
template <class R, bool AIN>
__global__ void __launch_bounds__(128, KfPseudoMinBlocks<R>::v) kf_pseudo(const Prob<R> P) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  const bool win = warp_interior(P.g, i, j, k);
  bool pin = false;
  if constexpr (sizeof(R) == 8)
    if (!win && P.pairs == 2) pin = warp_on_grid(P.g, i, j);
  if (i > P.g.np || j > P.g.mp) return;
  if (!win) {
    if constexpr (sizeof(R) == 8) {
      if (pin) {
        if (warp_unit_faces(P, i, j, k))
          pseudo_body<R, AIN, false, true, true, false, true, true>(P, i, j, k);
        else
          pseudo_body<R, AIN, false, false, true, false, true, true>(P, i, j, k);
        return;
      }
    }
    pseudo_body<R, AIN, false>(P, i, j, k);
  } else if constexpr (sizeof(R) == 8) {
    const bool unit = warp_unit_faces(P, i, j, k);
    if (P.pairs == 2) {
      if (unit)
        pseudo_body<R, AIN, true, true, true, false, true, true>(P, i, j, k);
      else
        pseudo_body<R, AIN, true, false, true, false, true, true>(P, i, j, k);
    } else {
      if (unit)
        pseudo_body<R, AIN, true, true>(P, i, j, k);
      else
        pseudo_body<R, AIN, true>(P, i, j, k);
    }
  } else {
    pseudo_body<R, AIN, true>(P, i, j, k);
  }
}
// Ratios of at least 1 are recorded as RATIO_CAP (lim_ratio): the reverse
// limiter's min3 selects neither form, and the reverse bounds kernel
// recomputes its quotients from the recorded extrema and fluxes.
template <class R, bool NONOS, bool FIRST, bool KEEP>
__global__ void __launch_bounds__(128, (KfMinBlocks<R, 12, 12>::v)) kf_bounds(const Prob<R> P) {
  chain_begin();
  if constexpr (NONOS && sizeof(R) == 8) {  // FP32: per-lane quotients are cheaper than the barriers
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z + 1;
    const bool win = warp_interior(P.g, i, j, k);
    const bool valid = i <= P.g.np && j <= P.g.mp;
    RatioOps<R> r{};
    if (valid) {
      if (!win)
        r = bounds_body<R, true, FIRST, KEEP, false, 2>(P, i, j, k);
      else if (warp_unit_cell(P, i, j, k))
        r = bounds_body<R, true, FIRST, KEEP, true, 2, true>(P, i, j, k);
      else
        r = bounds_body<R, true, FIRST, KEEP, true, 2>(P, i, j, k);
    }
    block_ratios(P, i, j, k, valid, r);
  } else {
#define B(IN, U) bounds_body<R, NONOS, FIRST, KEEP, IN, 1, U>(P, i, j, k)
    FCELL_U(B)
#undef B
  }
}
template <class R, bool NONOS>
__global__ void __launch_bounds__(128, (KfMinBlocks<R, 16, 16>::v)) kf_limit(const Prob<R> P) {
  chain_begin();
#define B(IN) limit_body<R, NONOS, IN>(P, i, j, k)
  FCELL(B)
#undef B
}
template <class R>
__global__ void __launch_bounds__(128) kf_update(const Prob<R> P) {
  chain_begin();
#define B(IN, U) update_body<R, false, IN, U>(P, i, j, k)
  FCELL_U(B)
#undef B
}
#undef FCELL
#undef FCELL_U

// The values of pass t: its input field, pseudo-velocities, ratios and
// extrema from the records; `a` selects the "a" velocities the pass's
// pseudo-velocity read (the previous pass's limited ones) or its own
// limited velocities (for the limiter's forward).
template <class R>
Prob<R> pass_prob(const Prob<R>& P, const AdjPlan<R>& A, int t, bool prev_w) {
  Prob<R> Q = P;
  Q.xant = A.x[t];
  Q.v1 = A.v[t][0];
  Q.v2 = A.v[t][1];
  Q.v3 = A.v[t][2];
  Q.cp = A.cp[t];
  Q.cn = A.cn[t];
  Q.mx = A.mx[t];
  Q.mn = A.mn[t];
  Q.q = A.q[t];
  Q.f1 = A.fns[t][0];  // standard form: the unlimited donor fluxes of the pass
  Q.f2 = A.fns[t][1];
  Q.f3 = A.fns[t][2];
  const int tw = prev_w ? (t > 0 ? t - 1 : 0) : t;
  Q.w1 = A.w[tw][0];
  Q.w2 = A.w[tw][1];
  Q.w3 = A.w[tw][2];
  return Q;
}

// The pair sums of a pass's input field in the standard form's accumulators lf,
// which the gauge form does not use, instead of the pass's cp, cn and q.
template <class R>
void pairs_in_lf(Prob<R>* Q, const AdjPlan<R>& A) {
  Q->cp = A.lf[0];
  Q->cn = A.lf[1];
  Q->q = A.lf[2];
}

// The forward records of one step (every pass's input field, velocities,
// ratios and extrema) into A's record arrays.  out: when given, the last
// pass's update also writes the step's output field there (interior cells),
// so that a checkpointed reverse sweep rebuilds a segment and records it in
// one pass.
//
// keep (FP64 gauge, one pass): the pair sums stay for the reverse that follows,
// the field's in lf, the velocities' in the workspace's f1..f3.
template <class R>
int record_passes(const Prob<R>& P, const AdjPlan<R>& A, int nonos, const Arr<R>* out, bool keep_pairs, cudaStream_t s) {
  const Geo& g = P.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  const int np_ = A.npass;
  const bool keep = np_ > 1;
  const size_t ncell = (size_t)g.np * g.mp * g.lp;
  int n = 0;
  Prob<R> F = P;
  F.xant = A.x[0];
  chain_launch(kf_upwind<R>, grd, blk, 0, s, F);
  n++;
  for (int t = 0; t < np_; t++) {
    Prob<R> Qa = pass_prob(P, A, t, true);
    // FP64 gauge: pair sums of the pass's input field into its cp/cn/q
    // records, which the bounds kernel fills afterwards, and the velocity
    // pairs into the workspace's f1..f3 (unused by the gauge form)
    Qa.pairs = (!P.stdf && sizeof(R) == 8) ? 2 : 0;
    if (Qa.pairs) {
      Qa.f1 = P.f1;
      Qa.f2 = P.f2;
      Qa.f3 = P.f3;
      if (keep_pairs) pairs_in_lf(&Qa, A);
      if (t == 0) chain_launch(kf_pairs<R, true, true>, grd, blk, 0, s, Qa);
      else chain_launch(kf_pairs<R, false, true>, grd, blk, 0, s, Qa);
      n++;
    }
    if (t == 0) chain_launch(kf_pseudo<R, true>, grd, blk, 0, s, Qa);
    else chain_launch(kf_pseudo<R, false>, grd, blk, 0, s, Qa);
    const Prob<R> Q = pass_prob(P, A, t, false);
    if (nonos && keep && t > 0) {  // the running extrema continue from the previous pass
      if (cudaMemcpyAsync(A.mx[t].p, A.mx[t - 1].p, ncell * sizeof(R), cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
          cudaMemcpyAsync(A.mn[t].p, A.mn[t - 1].p, ncell * sizeof(R), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
        return -5;
    }
    if (!nonos) chain_launch(kf_bounds<R, false, true, false>, grd, blk, 0, s, Q);
    else if (!keep) chain_launch(kf_bounds<R, true, true, false>, grd, blk, 0, s, Q);
    else if (t == 0) chain_launch(kf_bounds<R, true, true, true>, grd, blk, 0, s, Q);
    else chain_launch(kf_bounds<R, true, false, true>, grd, blk, 0, s, Q);
    n += 2;
    // only the update and the next pass read the limited velocities: the last
    // pass of a step whose output is not wanted leaves them out
    if (t == np_ - 1 && !out) break;
    // the limited fluxes (standard form) go to the workspace scratch: only
    // the update reads them
    Prob<R> L = Q;
    L.f1 = P.f1;
    L.f2 = P.f2;
    L.f3 = P.f3;
    if (nonos) chain_launch(kf_limit<R, true>, grd, blk, 0, s, L);
    else chain_launch(kf_limit<R, false>, grd, blk, 0, s, L);
    Prob<R> U = L;
    U.xant = t < np_ - 1 ? A.x[t + 1] : *out;
    chain_launch(kf_update<R>, grd, blk, 0, s, U);
    n += 2;
  }
  add_launches(n);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

int run_record_ratios(const Prob<float>& P, const AdjPlan<float>& A, cudaStream_t s) {
  const Geo& g = P.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  chain_launch(kf_bounds<float, true, true, false>, grd, blk, 0, s, pass_prob(P, A, 0, false));
  add_launches(1);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
int run_record_reciprocals(const Prob<float>& P, const AdjPlan<float>& A, cudaStream_t s) {
  const Geo& g = P.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  Prob<float> F = P;
  F.xant = A.x[0];  // the upwind field comes with them
  chain_launch(kf_upwind<float>, grd, blk, 0, s, F);
  add_launches(1);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <class R>
int run_step_record(const Prob<R>& P, const AdjPlan<R>& A, int nonos, const Arr<R>* out, cudaStream_t s) {
  return record_passes<R>(P, A, nonos, out, false, s);
}

// The reverse kernels of one recorded step: lambda of the step's output (A.lam)
// becomes lambda of its input; the velocity gradients accumulate into A.gu*.
// kept: the record's pair sums are where record_passes kept them.
template <class R>
int reverse_passes(const Prob<R>& P, const AdjPlan<R>& A, int nonos, bool kept, cudaStream_t s) {
  const Geo& g = P.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  const int np_ = A.npass;
  int n = 0;
  // The accumulators that kernels add to.  Standard form: all of them.  Gauge
  // form: lambda_w of every pass but the last (the next pass's pseudo-velocity
  // adds to it), and of the last where mass fluxes have cotangents; with the
  // limiter lcp and lcn, and the running extrema of every pass but the last.
  // Every other array is stored whole by the first kernel that writes it.
  const bool mass = A.rho && A.lm1.p;
  const size_t n1 = A.pass_acc_elems / 12;  // elements of one field
  auto zero = [&](R* p, size_t fields) { return cudaMemsetAsync(p, 0, fields * n1 * sizeof(R), s) == cudaSuccess; };
  if (P.stdf) {
    if (cudaMemsetAsync(A.acc, 0, A.acc_elems * sizeof(R), s) != cudaSuccess) return -5;
  } else {  // a pass's six: lx, lw*3, lmx, lmn
    for (int t = 0; t < np_ - 1; t++)
      if (!zero(A.acc + (6 * t + 1) * n1, 5)) return -5;
    if (mass && !zero(A.acc + (6 * (np_ - 1) + 1) * n1, 3)) return -5;
  }
  if (mass) {  // the density step's mass fluxes read the last pass's limited fluxes
    AdjArr<R> m{};
    m.lw1 = A.lw[np_ - 1][0];
    m.lw2 = A.lw[np_ - 1][1];
    m.lw3 = A.lw[np_ - 1][2];
    m.lm1 = A.lm1;
    m.lm2 = A.lm2;
    m.lm3 = A.lm3;
    chain_launch(ka_mass_to_w<R>, grd, blk, 0, s, P, m);
    n++;
  }
  // ---- reverse, last pass first
  for (int t = np_ - 1; t >= 0; t--) {
    if (P.stdf && t < np_ - 1 && !zero(A.pass_acc, 12)) return -5;
    if (!P.stdf && nonos && !zero(A.pass_acc + 3 * n1, 2)) return -5;  // lcp, lcn
    const Prob<R> Q = pass_prob(P, A, t, true);
    AdjArr<R> a{};
    a.lxant = A.lx[t];
    a.lv1 = A.lv[0];
    a.lv2 = A.lv[1];
    a.lv3 = A.lv[2];
    a.lw1 = A.lw[t][0];
    a.lw2 = A.lw[t][1];
    a.lw3 = A.lw[t][2];
    a.lcp = A.lcp;
    a.lcn = A.lcn;
    a.lx = A.lam;  // once the last pass's update has read the caller's lambda
    a.lam = t == np_ - 1 ? A.lam : A.lx[t + 1];
    a.gu1 = A.gu1;
    a.gu2 = A.gu2;
    a.gu3 = A.gu3;
    a.la1 = t == 0 ? A.gu1 : A.lw[t - 1][0];
    a.la2 = t == 0 ? A.gu2 : A.lw[t - 1][1];
    a.la3 = t == 0 ? A.gu3 : A.lw[t - 1][2];
    a.lmx = A.lmx[t];
    a.lmn = A.lmn[t];
    a.lmxp = A.lmx[t > 0 ? t - 1 : 0];
    a.lmnp = A.lmn[t > 0 ? t - 1 : 0];
    a.mxp = A.mx[t > 0 ? t - 1 : 0];
    a.mnp = A.mn[t > 0 ? t - 1 : 0];
    a.lg1 = A.lg[0];
    a.lg2 = A.lg[1];
    a.lg3 = A.lg[2];
    a.lf1 = A.lf[0];
    a.lf2 = A.lf[1];
    a.lf3 = A.lf[2];
    a.lq = A.lq;
    AdjArr<R> au = a;
    if (t < np_ - 1) au.lx.p = nullptr;
    if (P.stdf) {
      chain_launch(ka_update_std<R>, grd, blk, 0, s, Q, au);
      if (nonos) {
        chain_launch(ka_limit_std<R, true>, grd, blk, 0, s, Q, a);
        if (t == 0) chain_launch(ka_bounds<R, true, true>, grd, blk, 0, s, Q, a);
        else chain_launch(ka_bounds<R, false, true>, grd, blk, 0, s, Q, a);
        n++;
      } else {
        chain_launch(ka_limit_std<R, false>, grd, blk, 0, s, Q, a);
      }
      if (t == 0) chain_launch(ka_pseudo_std<R, true>, grd, blk, 0, s, Q, a);
      else chain_launch(ka_pseudo_std<R, false>, grd, blk, 0, s, Q, a);
    } else {
      if (t == np_ - 1) {  // nothing carried back, nothing added to lambda_w
        a.lmx.p = a.lmn.p = nullptr;
        if (!mass) a.lw1.p = a.lw2.p = a.lw3.p = nullptr;
      }
      chain_launch(ka_update<R>, grd, blk, 0, s, Q, au);
      if (nonos) {
        chain_launch(ka_limit<R, true>, grd, blk, 0, s, Q, a);
        if (t == 0) chain_launch(ka_bounds<R, true, false>, grd, blk, 0, s, Q, a);
        else chain_launch(ka_bounds<R, false, false>, grd, blk, 0, s, Q, a);
        n++;
      } else {
        chain_launch(ka_limit<R, false>, grd, blk, 0, s, Q, a);
      }
      // the pass's cp/cn/q records are dead once the reverse bounds ran:
      // they take the pair sums of its input field, and the workspace's
      // f1..f3 the velocity pairs
      Prob<R> Qp = Q;
      Qp.f1 = P.f1;
      Qp.f2 = P.f2;
      Qp.f3 = P.f3;
      if (kept) pairs_in_lf(&Qp, A);
      else if (t == 0) chain_launch(kf_pairs<R, true, true>, grd, blk, 0, s, Qp);
      else chain_launch(kf_pairs<R, false, true>, grd, blk, 0, s, Qp);
      n += kept ? 0 : 1;
      if (sizeof(R) == 4 && g.bx && g.by && g.bz) {
        if constexpr (sizeof(R) == 4) {
          if (t == 0) chain_launch(ka_cross<R, true>, grd, blk, 0, s, Qp, a);
          else chain_launch(ka_cross<R, false>, grd, blk, 0, s, Qp, a);
          chain_launch(ka_cross_sum<R>, grd, blk, 0, s, Qp, a);
          n++;
        }
      } else if (t == 0) {
        chain_launch(ka_pseudo<R, true>, grd, blk, 0, s, Qp, a);
      } else {
        chain_launch(ka_pseudo<R, false>, grd, blk, 0, s, Qp, a);
      }
    }
    n += 3;
  }
  AdjArr<R> a0{};
  a0.lxant = A.lx[0];
  a0.lx = A.lam;
  a0.gu1 = A.gu1;
  a0.gu2 = A.gu2;
  a0.gu3 = A.gu3;
  if (A.rho && A.lm1.p) {
    a0.lm1 = A.lm1;
    a0.lm2 = A.lm2;
    a0.lm3 = A.lm3;
    chain_launch(ka_upwind<R, true>, grd, blk, 0, s, P, a0);
  } else {
    chain_launch(ka_upwind<R>, grd, blk, 0, s, P, a0);
  }
  n++;
  add_launches(n);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <class R>
int run_step_reverse(const Prob<R>& P, const AdjPlan<R>& A, int nonos, cudaStream_t s) {
  return reverse_passes<R>(P, A, nonos, false, s);
}

// Record and reverse of one step.  With one pass in FP64 (gauge) the record's
// pair sums serve the reverse too: 57 us of 256x256x64 not spent again.
template <class R>
int run_step_adjoint(const Prob<R>& P, const AdjPlan<R>& A, int nonos, cudaStream_t s) {
  const bool keep = sizeof(R) == 8 && !P.stdf && A.npass == 1;
  const int rc = record_passes<R>(P, A, nonos, nullptr, keep, s);
  return rc ? rc : reverse_passes<R>(P, A, nonos, keep, s);
}

template <class R>
int run_rho_out_adjoint(const Prob<R>& P, const Arr<R>& out, const Arr<R>& lxc, const Arr<R>& lp1,
                        const Arr<R>& lp2, const Arr<R>& lrh, const Arr<R>& lam, const Arr<R>& g_xinc,
                        const Arr<R>& g_pexe, cudaStream_t s) {
  const Geo& g = P.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  chain_launch(ka_rho_out<R>, grd, blk, 0, s, P, out, lxc, lp1, lp2, lrh, lam, g_xinc, g_pexe);
  add_launches(1);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <class R>
int run_seed(const Prob<R>& P, const Arr<R>& psi, const Arr<R>& target, const Arr<R>& lam, cudaStream_t s) {
  const Geo& g = P.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  chain_launch(ka_seed<R>, grd, blk, 0, s, P, psi, target, lam);
  add_launches(1);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template int run_step_adjoint<double>(const Prob<double>&, const AdjPlan<double>&, int, cudaStream_t);
template int run_step_adjoint<float>(const Prob<float>&, const AdjPlan<float>&, int, cudaStream_t);
template int run_step_record<double>(const Prob<double>&, const AdjPlan<double>&, int, const Arr<double>*,
                                     cudaStream_t);
template int run_step_record<float>(const Prob<float>&, const AdjPlan<float>&, int, const Arr<float>*,
                                    cudaStream_t);
template int run_step_reverse<double>(const Prob<double>&, const AdjPlan<double>&, int, cudaStream_t);
template int run_step_reverse<float>(const Prob<float>&, const AdjPlan<float>&, int, cudaStream_t);
template int run_rho_out_adjoint<double>(const Prob<double>&, const Arr<double>&, const Arr<double>&,
                                         const Arr<double>&, const Arr<double>&, const Arr<double>&,
                                         const Arr<double>&, const Arr<double>&, const Arr<double>&, cudaStream_t);
template int run_rho_out_adjoint<float>(const Prob<float>&, const Arr<float>&, const Arr<float>&, const Arr<float>&,
                                        const Arr<float>&, const Arr<float>&, const Arr<float>&, const Arr<float>&,
                                        const Arr<float>&, cudaStream_t);
template int run_seed<double>(const Prob<double>&, const Arr<double>&, const Arr<double>&, const Arr<double>&, cudaStream_t);
template int run_seed<float>(const Prob<float>&, const Arr<float>&, const Arr<float>&, const Arr<float>&, cudaStream_t);

}  // namespace mpdata
