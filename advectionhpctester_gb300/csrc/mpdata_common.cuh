// Shared device-side definitions of the MPDATA step: grid geometry, array
// views over the reference's Fortran layout, boundary index maps and the
// MPDATA point operators (advection/src_algorithms/mpdataoperators.inc:50-96).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace mpdata {

// Launches a kernel so that it may start while the one before it in the stream
// drains: its blocks take the slots that the last wave leaves free and wait in
// chain_begin() until every block of that kernel is done and its writes are
// visible.  Saves the launch latency between the short kernels of a step; a
// launch that follows a copy, a memset or another library's kernel waits for it
// as usual.  Every kernel launched this way calls chain_begin() before it
// touches memory, so each one's end also implies the end of all before it.
// chained = false: an ordinary launch, after the end of the one before.
template <class... P, class... A>
inline void chain_launch_if(bool chained, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                            A&&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}
template <class... P, class... A>
inline void chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  chain_launch_if(true, kernel, grid, block, smem, s, std::forward<A>(args)...);
}
// The two halves: the following kernel may start; this one's inputs are there.
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_begin() {
  chain_trigger();
  chain_wait();
}

// Grid geometry and boundary flags (1 = periodic axis).
struct Geo {
  int np, mp, lp, ih;
  int bx, by, bz;
};

// View of a 3-D Fortran-ordered array; p points at the logical element
// (1,1,1), so halo elements sit at negative offsets inside the caller's
// allocation.  Indices are the reference's 1-based (i,j,k).  The strides are
// 32-bit (the host rejects grids whose planes, halos included, reach 2^31
// elements), so each term of an offset is one 32x32->64 multiply-add.
template <class R>
struct Arr {
  R* p;
  int sy, sz;
  __device__ __forceinline__ long off(int i, int j, int k) const {
    return (long)(i - 1) + (long)(j - 1) * sy + (long)(k - 1) * sz;
  }
  __device__ __forceinline__ R ld(int i, int j, int k) const { return p[off(i, j, k)]; }
  __device__ __forceinline__ R& at(int i, int j, int k) const { return p[off(i, j, k)]; }
};

// Caller arrays with halo width ih: extents (n0, n1, *) along x and y.
template <class R>
inline Arr<R> caller_view(R* base, int ih, int n0, int n1) {
  const long sy = n0, sz = (long)n0 * n1;
  return Arr<R>{base + ih + ih * sy + ih * sz, (int)sy, (int)sz};
}
// Workspace scratch: interior cells (or faces 1..n along the own axis), no halo.
template <class R>
inline Arr<R> scratch_view(R* base, const Geo& g) {
  return Arr<R>{base, g.np, (int)((long)g.np * g.mp)};
}

// ---- index maps for reads one cell outside [1, n] ----
__device__ __forceinline__ int wrapi(int i, int n) { return i < 1 ? i + n : (i > n ? i - n : i); }
// reflection about the first/last interior cell: x(0)=x(2), x(n+1)=x(n-1)
// (cp_scnd_last_to_halo_xy_fulld, mpdataoperators.inc:479-513)
__device__ __forceinline__ int refl(int i, int n) { return i < 1 ? 2 - i : (i > n ? 2 * n - i : i); }
// zero gradient: x(0)=x(1), x(n+1)=x(n) (cp_last_to_halo_xy, mpdataoperators.inc:551-584)
__device__ __forceinline__ int clampi(int i, int n) { return i < 1 ? 1 : (i > n ? n : i); }

// ---- order-preserving selects -------------------------------------------
// On GB300 every FP64 compare, min and max issues on the FP64 pipe, which
// retires about 2 operations per SM per clock, while the integer pipe retires
// about 64.  For doubles these selects therefore work on the bit patterns:
// the order key of x is its bits with the magnitude bits flipped when the
// sign is set, so signed 64-bit order of keys is IEEE order of values, except
// that -0 orders below +0 and a NaN orders beyond the infinities.  The
// selects below return what the reference's compare-and-select returns, bit
// for bit, and use the keys alone where the two orders agree.  Float keeps the
// native FP32 compares (cheap on the FP32/ALU pipes).
__device__ __forceinline__ long long okey(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double from_okey(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
__device__ __forceinline__ bool sgn(double y) { return __double2hiint(y) < 0; }
__device__ __forceinline__ bool sgn(float y) { return __float_as_int(y) < 0; }

// -y and y != 0 as integer operations on the two 32-bit halves.  Written in
// PTX so that the compiler cannot turn them back into an FP64 negation (a
// DADD) or an FP64 compare (a DSETP), both of which issue on the FP64 pipe.
// IEEE negation is exactly a flip of the sign bit.
__device__ __forceinline__ double neg_bits(double y) {
  double r;
  asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\txor.b32 hi, hi, 0x80000000;\n\t"
      "mov.b64 %0, {lo, hi};\n\t}"
      : "=d"(r)
      : "d"(y));
  return r;
}
__device__ __forceinline__ bool nonzero_bits(double y) {
  unsigned lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(y));
  return ((hi << 1) | lo) != 0u;
}

// Products by a power of two 2^-s on the integer pipe.  When x is a normal
// number whose exponent field e satisfies s < e < 0x7FF, x*2^-s is a normal
// number with the same significand and e-s as its exponent field: the FP64
// multiplication rounds nothing there, so lowering the field gives its bits.
// A zero keeps its sign (0*2^-s = 0).  Subnormal results and subnormal,
// infinite or NaN operands take the multiplication itself, behind a call so
// that it is branched around.  Float multiplies (its pipe is not the bound).
static __device__ __noinline__ double mul_call(double x, double y) { return x * y; }
__device__ __forceinline__ double scale_down(double x, int s, double k) {  // k = 2^-s, 1 <= s <= 60
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7FFu;
  if (e - (unsigned)(s + 1) < (unsigned)(0x7FE - s)) return __hiloint2double(hi - (s << 20), lo);
  if ((((unsigned)hi << 1) | (unsigned)lo) == 0u) return x;
  return mul_call(x, k);
}
template <int S>
__device__ __forceinline__ double scale_down(double x) {
  return scale_down(x, S, 1.0 / (double)(1LL << S));
}
template <int S>
__device__ __forceinline__ float scale_down(float x) {
  return x * (1.0f / (float)(1 << S));
}
// Products by 2^S the same way: a normal x whose exponent field e satisfies
// e + S < 0x7FF gains S in the field; zeros pass, everything else multiplies.
template <int S>
__device__ __forceinline__ double scale_up(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7FFu;
  if (e - 1u < (unsigned)(0x7FE - S)) return __hiloint2double(hi + (S << 20), lo);
  if ((((unsigned)hi << 1) | (unsigned)lo) == 0u) return x;
  return mul_call(x, (double)(1LL << S));
}
template <int S>
__device__ __forceinline__ float scale_up(float x) {
  return x * (float)(1 << S);
}

// pp(y) = max(0,y), pn(y) = -min(0,y)  (mpdataoperators.inc:50-59)
__device__ __forceinline__ double pp(double y) { return sgn(y) ? 0.0 : y; }
__device__ __forceinline__ double pn(double y) { return sgn(y) ? neg_bits(y) : 0.0; }
// FP32: one max instruction each.  PTX max.f32 orders -0 below +0 and
// returns the other operand for a NaN, so max(y, +0) is y > 0 ? y : +0 and
// max(-y, +0) is y < 0 ? -y : +0 for every y, zeros and NaNs included.
__device__ __forceinline__ float fmax0(float y) {
  float r;
  asm("max.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(y));
  return r;
}
__device__ __forceinline__ float pp(float y) { return fmax0(y); }
__device__ __forceinline__ float pn(float y) { return fmax0(-y); }
// a > b as the FP64 compare gives it, on the integer pipe: false when either
// operand is a NaN or both are zeros (+0 == -0), else the order of the keys.
__device__ __forceinline__ bool ieee_gt(double a, double b) {
  const unsigned long long ka = (unsigned long long)__double_as_longlong(a) << 1,
                           kb = (unsigned long long)__double_as_longlong(b) << 1;  // magnitudes, doubled
  const unsigned long long inf2 = 0xFFE0000000000000ULL;
  if (ka > inf2 || kb > inf2 || (ka | kb) == 0ULL) return false;
  return okey(a) > okey(b);
}
// The reference's compare-and-select max and min (a > b ? a : b, a < b ?
// a : b): ties and NaNs keep the second operand.
__device__ __forceinline__ double mx2(double a, double b) { return ieee_gt(a, b) ? a : b; }
__device__ __forceinline__ double mn2(double a, double b) { return ieee_gt(b, a) ? a : b; }
__device__ __forceinline__ float mx2(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float mn2(float a, float b) { return a < b ? a : b; }
// The same selects in the order of the keys alone, which differs from them
// only when both operands are zeros of opposite signs (-0 orders below +0) or
// an operand is a NaN.
__device__ __forceinline__ double mx2k(double a, double b) { return okey(a) > okey(b) ? a : b; }
__device__ __forceinline__ double mn2k(double a, double b) { return okey(a) < okey(b) ? a : b; }
// A test of the high word that holds for every zero and NaN (the extrema
// the key order may pick differently): x is a zero, an infinity, a NaN, or a
// subnormal number whose high word has no significand bit (|x| < 2^-1042).
__device__ __forceinline__ bool zero_nan_hi(double x) {
  return ((unsigned)__double2hiint(x) & 0x7FFFFFFFu) - 1u >= 0x7FEFFFFFu;
}

// Running max and min over a set of values (the limiter's 7-point stars), in
// key order for doubles: exact whenever the extremum found is neither a zero
// nor a NaN (it is then the one value of its bits in the set).
template <class R> struct Extrema;
template <> struct Extrema<double> {
  long long kx, kn;
  __device__ __forceinline__ explicit Extrema(double v) { kx = kn = okey(v); }
  __device__ __forceinline__ void add(double v) {
    const long long k = okey(v);
    kx = k > kx ? k : kx;
    kn = k < kn ? k : kn;
  }
  __device__ __forceinline__ double max() const { return from_okey(kx); }
  __device__ __forceinline__ double min() const { return from_okey(kn); }
};
template <> struct Extrema<float> {
  float x, n;
  __device__ __forceinline__ explicit Extrema(float v) : x(v), n(v) {}
  __device__ __forceinline__ void add(float v) { x = v > x ? v : x; n = v < n ? v : n; }
  __device__ __forceinline__ float max() const { return x; }
  __device__ __forceinline__ float min() const { return n; }
};

// Correctly rounded FP64 quotient on the integer and FP32 pipes.  On GB300 an
// IEEE division holds the FP64 pipe for about nine of its instructions (64 G/s
// for the whole chip), which bound every kernel that divides; the integer
// pipes beside it are mostly idle.  This is a long division in two 26/27-bit
// digits with exact remainders (very high radix division with a short
// reciprocal: Wong and Flynn, IEEE Trans. Computers 41(8), 1992), written from
// the mathematics:
//   N, D in [2^52, 2^53) are the significands, N doubled when N < D, so that
//   N/D lies in [1, 2).  R = 2^83/D less up to 2 units, never more: MUFU.RCP of
//   D's leading 24 bits (within 1 ulp) and one correction from its residual,
//   whose own error is below 2^-14 of a unit.  A digit floor(rem*R) is then at
//   most one too small (it loses less than 0.7 of a unit), so that a remainder
//   stays in [0, 2D) and is exact modulo 2^64; the last comparison with D
//   settles the 53 fraction bits, the last of which rounds: a quotient of two
//   53-bit numbers is never exactly between two others.
// Exponents within 500 of the bias keep the result normal; zeros over such a
// denominator are their own quotient; everything else takes the instruction
// sequence of the compiler, behind a call.  About 60 integer and FP32
// instructions: the standard form's nine quotients per cell and pass went from
// 1.02 to 0.66 ms per step at 191x157x61 with a varying density (64x64x32, unit
// density: 100 to 68 us), the density step at 160x129x48 from 414 to 340 us.
static __device__ __noinline__ double div_hw(double x, double r) { return x / r; }
__device__ __forceinline__ double quot_int(unsigned nh, unsigned nl, unsigned dh, unsigned dl) {
  const unsigned Nh = (nh & 0xFFFFFu) | 0x100000u, Dh = (dh & 0xFFFFFu) | 0x100000u;
  unsigned long long N = ((unsigned long long)Nh << 32) | nl;
  const unsigned long long D = ((unsigned long long)Dh << 32) | dl;
  const bool lt = N < D;
  if (lt) N <<= 1;
  const float df = __uint_as_float((__funnelshift_l(dl, dh, 3) & 0x7FFFFFu) | 0x3F800000u);
  const float lo = __uint2float_rz(dl & 0x1FFFFFFFu);  // D = 2^52*df + lo
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(df));
  float e = __fmaf_rn(-df, r0, 1.0f);
  e = __fmaf_rn(-lo, r0 * 2.220446049250313e-16f, e);
  const float c = __fmaf_rn(e * r0, 2147483648.0f, -0.0625f);
  const unsigned R = __float2uint_rz(r0 * 2147483648.0f) + (unsigned)__float2int_rd(c);
  const unsigned t1 = __umulhi((unsigned)(N >> 22), R) >> 2;
  const unsigned long long r1 = (N << 27) - (unsigned long long)t1 * D;
  const unsigned t2 = __umulhi((unsigned)(r1 >> 22), R) >> 3;
  const unsigned long long r2 = (r1 << 26) - (unsigned long long)t2 * D;
  unsigned long long q = ((unsigned long long)t1 << 26) + t2 + (r2 >= D ? 2ULL : 1ULL);
  q >>= 1;
  const unsigned eh = (nh & 0x7FF00000u) - (dh & 0x7FF00000u) + 0x3FE00000u - (lt ? 0x100000u : 0u);
  const unsigned qh = ((unsigned)(q >> 32) + eh) | ((nh ^ dh) & 0x80000000u);
  return __hiloint2double((int)qh, (int)(unsigned)q);
}
__device__ __forceinline__ double quot(double n, double d) {
  const unsigned nh = (unsigned)__double2hiint(n), nl = (unsigned)__double2loint(n);
  const unsigned dh = (unsigned)__double2hiint(d), dl = (unsigned)__double2loint(d);
  constexpr unsigned lo = (1023u - 500u) << 20, span = 1000u << 20;
  const unsigned en = (nh & 0x7FF00000u) - lo, ed = (dh & 0x7FF00000u) - lo;
  if ((en > ed ? en : ed) < span) return quot_int(nh, nl, dh, dl);
  if (((nh << 1) | nl) == 0u && ed < span) return __hiloint2double((int)((nh ^ dh) & 0x80000000u), 0);
  return div_hw(n, d);
}
__device__ __forceinline__ float quot(float n, float d) { return n / d; }

// Unit densities.  x*1 == x, x/1 == x, 1/1 == 1 and 2/(1+1) == 1 hold
// exactly in IEEE arithmetic (signed zeros and infinities included), so when a
// density or its reciprocal is exactly 1 these operations are skipped and no
// bit of any result changes.  The test is an integer compare of the bit
// pattern.  Unit densities are the reference test driver's setting
// (init_data: h = rhr = 1); on GB300 an FP64 division costs ~9 FP64
// instructions.
// FP64 only: an FP32 division or multiply costs less than the test on the
// FP32 kernels, which are bound by instruction issue.  The FP64 division sits
// behind a call so that it is branched around, not evaluated and discarded.
__device__ __forceinline__ bool is_one(double r) { return __double_as_longlong(r) == 0x3FF0000000000000LL; }
static __device__ __noinline__ double div_call(double x, double r) { return quot(x, r); }
__device__ __forceinline__ double mul1(double x, double r) { return is_one(r) ? x : x * r; }
__device__ __forceinline__ double div1(double x, double r) { return is_one(r) ? x : div_call(x, r); }
__device__ __forceinline__ double rcp1(double r) { return is_one(r) ? 1.0 : div_call(1.0, r); }
__device__ __forceinline__ float mul1(float x, float r) { return x * r; }
__device__ __forceinline__ float div1(float x, float r) { return x / r; }
__device__ __forceinline__ float rcp1(float r) { return 1.0f / r; }

// Limiter ratio n/d (n >= 0, d >= ep > 0) whose readers take min(1, n/d, ...):
// when n >= d and d is finite the IEEE quotient is >= 1, and RATIO_CAP = 2 is
// returned without dividing.  The forward minimum is 1 either way, bit for
// bit; the adjoint's min3 never selects a ratio above 1, which is the
// derivative of any quotient above 1 (a quotient of exactly 1, a tie with the
// constant, is the one case whose subgradient it picks differently).  NaN
// operands (n above +Inf, d not a positive finite number) divide as usual.
// The test runs on the integer pipe: for non-negative numbers the bit
// patterns order as the values do.
__device__ __forceinline__ bool ratio_ge1(double n, double d) {
  const long long nb = __double_as_longlong(n), db = __double_as_longlong(d), inf = 0x7FF0000000000000LL;
  return db > 0 && db < inf && nb >= db && nb <= inf;
}
constexpr int RATIO_CAP = 2;
__device__ __forceinline__ double lim_ratio(double n, double d) {
  return ratio_ge1(n, d) ? double(RATIO_CAP) : div_call(n, d);
}
// n/d is n itself when n is a zero and d a positive finite number (IEEE
// 0/d is a zero with the sign of n).  A field on an exactly zero background
// has two such ratios at every background cell, where x equals its star's
// minimum and maximum.
__device__ __forceinline__ bool ratio_zero(double n, double d) {
  const long long db = __double_as_longlong(d), inf = 0x7FF0000000000000LL;
  return ((unsigned long long)__double_as_longlong(n) << 1) == 0ULL && db > 0 && db < inf;
}
// FP32: d in (0, +Inf) as bits [1, 0x7F7FFFFF] and n in [d, +Inf] as bits,
// each one unsigned range test (n with its sign bit set fails the second).
__device__ __forceinline__ bool ratio_ge1(float n, float d) {
  const unsigned nb = __float_as_uint(n), db = __float_as_uint(d);
  return db - 1u < 0x7F7FFFFFu && nb - db <= 0x7F800000u - db;
}
__device__ __forceinline__ float lim_ratio(float n, float d) { return ratio_ge1(n, d) ? float(RATIO_CAP) : n / d; }

// ---- point operators (device forms of mpdataoperators.inc:50-96) ----
__device__ __forceinline__ float donor(float y1, float y2, float a) { return pp(a) * y1 - pn(a) * y2; }
// FP64 donor flux pp(a)*y1 - pn(a)*y2 with one multiplication.  For finite
// operands one of the two products is a zero, and rounding is symmetric in
// sign, so a nonzero result is a*y1 (a > 0) or -((-a)*y2) = a*y2 (a <= 0).
// When that product is zero, the two signed zeros the reference subtracts
// give -0 exactly when y1's sign bit is set and y2's is not, whatever a is;
// that zero is returned.  The tests are integer operations, which leave the
// FP64 pipe (the bound of every FP64 stage) to the multiplication.
__device__ __forceinline__ double donor(double y1, double y2, double a) {
  const double m = a * (__double_as_longlong(a) > 0 ? y1 : y2);
  if (nonzero_bits(m)) return m;
  return (sgn(y1) && !sgn(y2)) ? -0.0 : 0.0;
}
template <class R> __device__ __forceinline__ R vdyf(R x1, R x2, R a, R rinv) {
  return scale_down<1>((fabs(a) - mul1(a * a, rinv)) * (x2 - x1));
}
template <class R> __device__ __forceinline__ R rat4(R z0, R z1, R z2, R z3) {
  return scale_down<2>((z3 + z2) - (z1 + z0));
}
template <class R> __device__ __forceinline__ R vdyfa(R x1, R x2, R a, R rinv, R ep) {
  return quot((fabs(a) - mul1(a * a, rinv)) * (fabs(x2) - fabs(x1)), fabs(x2) + fabs(x1) + ep);
}
template <class R> __device__ __forceinline__ R vcorra(R a, R b, R y1, R y2, R rinv) {
  return -quot(mul1(scale_down<3>(a) * b * y1, rinv), y2);
}
// Forms of the pseudo-velocity operators for the stage kernels.  U: every face
// density of the warp is exactly 1, so the products by it are dropped (exact,
// as above).  dif4 is rat4 without its factor 0.25, which the caller folds into
// the 0.125 of the cross term (0.125*0.25 = 0.03125).  Scaling by a power of
// two commutes with rounding, so the folded form gives the same bits as
// rat4's order whenever no intermediate is subnormal (|value| < 2^-1022 in
// FP64, 2^-126 in FP32), and differs by at most a subnormal ulp otherwise.
template <bool U, class R> __device__ __forceinline__ R hmul(R x, R hm) { return U ? x : x * hm; }
template <bool U, class R> __device__ __forceinline__ R vdyf_u(R x1, R x2, R a, R hm) {
  return scale_down<1>((fabs(a) - hmul<U>(a * a, hm)) * (x2 - x1));
}
template <bool U, class R> __device__ __forceinline__ R vdyfa_u(R x1, R x2, R a, R hm, R ep) {
  return quot((fabs(a) - hmul<U>(a * a, hm)) * (fabs(x2) - fabs(x1)), fabs(x2) + fabs(x1) + ep);
}
// vdyfa_u with |x1|+|x2| at hand (sum)
template <bool U, class R> __device__ __forceinline__ R vdyfa_s(R x1, R x2, R a, R hm, R sum, R ep) {
  return quot((fabs(a) - hmul<U>(a * a, hm)) * (fabs(x2) - fabs(x1)), sum + ep);
}
template <bool U, class R> __device__ __forceinline__ R vcorra_u(R a, R b, R y1, R y2, R hm) {
  return -quot(hmul<U>(scale_down<3>(a) * b * y1, hm), y2);
}
template <class R> __device__ __forceinline__ R dif4(R z0, R z1, R z2, R z3) { return (z3 + z2) - (z1 + z0); }
template <class R> __device__ __forceinline__ R possign(R x) { return sgn(x) ? R(0) : R(1); }
// min3(a, b) = mn2(mn2(1, a), b).  For doubles whose high words are both
// below 0x7FF00000 (non-negative, finite: the limiter's ratios) the raw bit
// patterns order as the values do, +0 included, so two integer compares give
// the result; anything else (a sign bit, an infinity, a NaN) takes the
// compares' own semantics.
__device__ __forceinline__ float min3(float a, float b) { return mn2(mn2(1.0f, a), b); }
static __device__ __noinline__ double min3_exact(double a, double b) { return mn2(mn2(1.0, a), b); }
__device__ __forceinline__ double min3(double a, double b) {
  const unsigned ha = (unsigned)__double2hiint(a), hb = (unsigned)__double2hiint(b);
  if ((ha > hb ? ha : hb) < 0x7FF00000u) {
    const long long ba = __double_as_longlong(a), bb = __double_as_longlong(b), one = 0x3FF0000000000000LL;
    const long long t = one < ba ? one : ba;
    return __longlong_as_double(t < bb ? t : bb);
  }
  return min3_exact(a, b);
}
// 1/(0.5*(h1+h2)) == 2/(h1+h2) exactly: the halving is an exact scaling.
__device__ __forceinline__ double rhm(double h1, double h2) {
  return is_one(h1) && is_one(h2) ? 1.0 : div_call(2.0, h1 + h2);
}
__device__ __forceinline__ float rhm(float h1, float h2) { return 2.0f / (h1 + h2); }

// ep_nonos (common/epsilons.f90:3)
template <class R> struct Eps;
template <> struct Eps<double> { static constexpr double v = 1e-10; };
template <> struct Eps<float> { static constexpr float v = 1e-10f; };

}  // namespace mpdata
