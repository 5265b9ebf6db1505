// Single-problem launch sequence of the MPDATA step (strict-IEEE path).
//
// One kernel per stage of the reference's antidiffusive iteration, one thread
// per cell, every face quantity computed exactly once (the reference
// recomputes shared faces per cell).  The per-cell arithmetic lives in
// mpdata_body.cuh.  Built with --fmad=false and IEEE division, so results are
// bit-identical to a strict-IEEE CPU evaluation of the reference's
// expressions (up to the sign of zero).
#include "mpdata_body.cuh"
#include "mpdata_stages.cuh"

namespace mpdata {

#define CELL_INDEX                                          \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1; \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1; \
  const int k = blockIdx.z + 1;                             \
  if (i > P.g.np || j > P.g.mp) return;

// Interior warps take the body without boundary maps (IN = true).
#define CELL_DISPATCH(BODY)                                 \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1; \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1; \
  const int k = blockIdx.z + 1;                             \
  const bool win = warp_interior(P.g, i, j, k);             \
  if (i > P.g.np || j > P.g.mp) return;                     \
  if (win) {                                                \
    BODY(true);                                             \
  } else {                                                  \
    BODY(false);                                            \
  }

// As CELL_DISPATCH, with the unit-density instantiation (BODY(IN, U)) for
// interior warps whose densities are all exactly 1.
#define CELL_DISPATCH_U(BODY)                               \
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1; \
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1; \
  const int k = blockIdx.z + 1;                             \
  const bool win = warp_interior(P.g, i, j, k);             \
  if (i > P.g.np || j > P.g.mp) return;                     \
  if (!win) {                                               \
    BODY(false, false);                                     \
  } else if (warp_unit_cell(P, i, j, k)) {                  \
    BODY(true, true);                                       \
  } else {                                                  \
    BODY(true, false);                                      \
  }

// Minimum resident 128-thread blocks per SM asked of the register allocator
// for the upwind, limiter-bounds and limited-flux kernels.  An explicit bound
// is always given: with none, or with 1, ptxas allots these kernels far more
// registers (k_limit 32 -> 56, k_upwind 48 -> 78 in FP32) and they run
// slower.  FP64 values from a sweep at 512x512x128 (upwind 8: -3%, bounds 12:
// -13% with a 12-byte spill, limit 16: -7%); FP32 from a sweep too (upwind
// 12: -12%, bounds 16: -4%, limit 16 and pseudo 8 as they were).
// Build-time overridable for tuning sweeps.
#ifndef MPDATA_MINB_UPWIND_F64
#define MPDATA_MINB_UPWIND_F64 8
#endif
#ifndef MPDATA_MINB_BOUNDS_F64
#define MPDATA_MINB_BOUNDS_F64 12
#endif
#ifndef MPDATA_MINB_LIMIT_F64
#define MPDATA_MINB_LIMIT_F64 16
#endif
#ifndef MPDATA_MINB_UPWIND_F32
#define MPDATA_MINB_UPWIND_F32 12
#endif
#ifndef MPDATA_MINB_BOUNDS_F32
#define MPDATA_MINB_BOUNDS_F32 16
#endif
#ifndef MPDATA_MINB_LIMIT_F32
#define MPDATA_MINB_LIMIT_F32 16
#endif
template <class R, int N64, int N32>
struct MinBlocks {
  static constexpr int v = sizeof(R) == 8 ? N64 : N32;
};

template <class R, bool ANTIDIFF>
__global__ void __launch_bounds__(128, (MinBlocks<R, MPDATA_MINB_UPWIND_F64, MPDATA_MINB_UPWIND_F32>::v)) k_upwind(const Prob<R> P) {
  if (P.chained) chain_begin();
#define B(IN, U) upwind_body<R, ANTIDIFF, true, IN, U>(P, i, j, k)
  CELL_DISPATCH_U(B)
#undef B
}
template <class R>
__global__ void __launch_bounds__(128) k_copy(const Prob<R> P) {
  if (P.chained) chain_begin();
  CELL_INDEX
  copy_body<R>(P, i, j, k);
}
// Minimum resident 128-thread blocks per SM asked of the register allocator
// for the pseudo-velocity kernel, whose interior path keeps ~60 neighbour
// loads in flight: FP32 is latency-bound and gains from 8 blocks (64
// registers, a 12-byte spill); FP64 takes 7 (72 registers, an 8-byte spill),
// which measured 5.02 ms per headline step at 512x512x128 against 5.32 with
// 5 blocks (88 registers) and 5.06 with 6 (80): the FP64 pipe waits on its
// loads (8 long-scoreboard stalls per issue at 5 blocks).  Build-time
// overridable for tuning sweeps.
#ifndef MPDATA_MINB_PSEUDO_F32
#define MPDATA_MINB_PSEUDO_F32 8
#endif
#ifndef MPDATA_MINB_PSEUDO_F64
#define MPDATA_MINB_PSEUDO_F64 7
#endif
template <class R>
struct PseudoMinBlocks {
  static constexpr int v = sizeof(R) == 4 ? MPDATA_MINB_PSEUDO_F32 : MPDATA_MINB_PSEUDO_F64;
};
// Whether the pseudo-velocity kernel issues every load before its stores
// (DEFER, see limit_form) or stores each face at once (fewer registers).
// FP64 measured the same either way, with 5 to 7 resident blocks (the FP64
// pipe is the bound); FP32 gains from DEFER.
#ifndef MPDATA_DEFER_PSEUDO_F64
#define MPDATA_DEFER_PSEUDO_F64 1
#endif
#ifndef MPDATA_DEFER_PSEUDO_F32
#define MPDATA_DEFER_PSEUDO_F32 1
#endif
template <class R>
struct PseudoDefer {
  static constexpr bool v = sizeof(R) == 4 ? MPDATA_DEFER_PSEUDO_F32 : MPDATA_DEFER_PSEUDO_F64;
};

template <class R, bool AIN>
__global__ void __launch_bounds__(128, PseudoMinBlocks<R>::v) k_pseudo(const Prob<R> P) {
  if (P.chained) chain_begin();
  constexpr bool D = PseudoDefer<R>::v;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  const bool win = warp_interior(P.g, i, j, k);
  const bool valid = i <= P.g.np && j <= P.g.mp;
  const unsigned act = __ballot_sync(0xffffffffu, valid);
  if (!valid) return;
  if constexpr (sizeof(R) == 8) {
    // every warp reads the stored pair sums, those at a boundary through the
    // boundary maps; the velocity pairs too where they are stored (pairs 2)
    const bool unit = warp_unit_faces(P, i, j, k, act);
    if (win) {
      if (P.pairs == 2) {
        if (unit)
          pseudo_body<R, AIN, true, true, true, false, D, true>(P, i, j, k);
        else
          pseudo_body<R, AIN, true, false, true, false, D, true>(P, i, j, k);
      } else {
        if (unit)
          pseudo_body<R, AIN, true, true, true, false, D>(P, i, j, k);
        else
          pseudo_body<R, AIN, true, false, true, false, D>(P, i, j, k);
      }
    } else if (P.pairs == 2) {
      if (unit)
        pseudo_body<R, AIN, false, true, true, false, D, true>(P, i, j, k);
      else
        pseudo_body<R, AIN, false, false, true, false, D, true>(P, i, j, k);
    } else {
      pseudo_body<R, AIN, false, false, true, false, D>(P, i, j, k);
    }
  } else if (win) {
    pseudo_body<R, AIN, true, false, false, false, D>(P, i, j, k);
  } else {
    pseudo_body<R, AIN, false, false, false, false, D>(P, i, j, k);
  }
}

template <class R, bool AIN, bool PV, bool STD>
__global__ void __launch_bounds__(128) k_pairs(const Prob<R> P) {
  if (P.chained) chain_begin();
  CELL_INDEX
  pairs_body<R, AIN, PV, STD>(P, i, j, k);
}
template <class R, bool NONOS, bool FIRST, bool KEEP>
__global__ void __launch_bounds__(128, (MinBlocks<R, MPDATA_MINB_BOUNDS_F64, MPDATA_MINB_BOUNDS_F32>::v)) k_bounds(const Prob<R> P) {
  if (P.chained) chain_begin();
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
    CELL_DISPATCH_U(B)
#undef B
  }
}
template <class R, bool NONOS>
__global__ void __launch_bounds__(128, (MinBlocks<R, MPDATA_MINB_LIMIT_F64, MPDATA_MINB_LIMIT_F32>::v)) k_limit(const Prob<R> P) {
  if (P.chained) chain_begin();
#define B(IN) limit_body<R, NONOS, IN>(P, i, j, k)
  CELL_DISPATCH(B)
#undef B
}
template <class R, bool LAST>
__global__ void __launch_bounds__(128) k_update(const Prob<R> P) {
  if (P.chained) chain_begin();
#define B(IN, U) update_body<R, LAST, IN, U>(P, i, j, k)
  CELL_DISPATCH_U(B)
#undef B
}

template <class R, bool LINER>
__global__ void __launch_bounds__(128) k_rho_out(const Prob<R> P) {
  if (P.chained) chain_begin();
  CELL_INDEX
  rho_out_body<R, LINER>(P, i, j, k);
}

// SMs of the current device (queried once; without a device those of the GB300 that the
// dispatch rules were measured on).
int num_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0)
      return v;
    cudaGetLastError();
    return 152;
  }();
  return n;
}

// ---- launch accounting ---------------------------------------------------
static unsigned long long g_launches = 0;
unsigned long long launch_count() { return __atomic_load_n(&g_launches, __ATOMIC_RELAXED); }
void add_launches(int n) { __atomic_add_fetch(&g_launches, (unsigned long long)n, __ATOMIC_RELAXED); }

// launch wrapper: optional event pair around the kernel, launch accounting
#define LAUNCH(stage, ...)                   \
  do {                                       \
    if (prof) prof->begin(stage, s);         \
    __VA_ARGS__;                             \
    if (prof) prof->end(stage, s);           \
    add_launches(1);                         \
  } while (0)

// Whether a step's kernels follow one another without the launch gap
// (chain_launch_if); blocks: of one kernel.  It saves two or three microseconds a
// kernel, 10 to 30% of a small step.  It costs where long kernels are bound by memory:
// the next one's blocks start as the last ones end, in another order over the SMs
// and their L2 halves (FP32 upwind step on 255x193x65, 25480 blocks: 51.7 us plain,
// 59.4 chained; 512x512x128 434 and 585; limiter off 0.87 of the chained time there;
// 128x128x64, 8192 blocks: 1.06 to 1.11).  And where an FP64 grid has one to four
// blocks an SM: the waiting blocks pile up on the SMs whose own end first, and the
// FP64 pipes of the others idle (gauge step on 32^3, 256 blocks: 40.4 us plain, 48.7
// chained; standard form 45.4 and 59.9; 33^3, 594 blocks: 47.3 and 50.0; but 24^3, 144
// blocks: 35.9 and 32.8; 40^3, 800 blocks: 1.04 to 1.12 of the chained time).
// The FP32 density step, whose predictor runs before it, keeps 3 to 5% of its chain.
bool chain_pays(long blocks, bool f64, int iord, bool limited_or_std, bool rho) {
  if (iord < 2 || !(f64 || rho)) return blocks <= 12000;
  if (!f64) return true;
  return !(limited_or_std && blocks >= 210 && blocks <= 700);
}

template <class R>
int run_step(const Prob<R>& P0, int iord, int nonos, Prof* prof, cudaStream_t s) {
  const Geo& g = P0.g;
  const dim3 blk(32, 4, 1);
  const dim3 grd((g.np + 31) / 32, (g.mp + 3) / 4, g.lp);
  Prob<R> P = P0;
  P.chained = chain_pays((long)grd.x * grd.y * grd.z, sizeof(R) == 8, iord, nonos || P.stdf, P.rho);
  if (iord < 2) {
    LAUNCH(ST_UPWIND, (chain_launch_if(P.chained, k_upwind<R, false>, grd, blk, 0, s, P)));
    if (P.rho) LAUNCH(ST_RHO_OUT, (chain_launch_if(P.chained, k_rho_out<R, true>, grd, blk, 0, s, P)));
    else LAUNCH(ST_COPY, (chain_launch_if(P.chained, k_copy<R>, grd, blk, 0, s, P)));
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  LAUNCH(ST_UPWIND, (chain_launch_if(P.chained, k_upwind<R, true>, grd, blk, 0, s, P)));
  const bool keep = iord > 2;
  // FP64: the pseudo-velocity stage reads precomputed pair sums of xant (pairs 1)
  // and, where three fields are free for them, of the pass velocities too (pairs
  // 2): not in the density step, whose upwind fluxes hold f1..f3, and in the
  // standard form in the first pass alone, whose w1..w3 are not yet written.  The
  // standard form went from 102 to 75 FP64 additions and products per cell and pass.
  Prob<R> Q = P;
  for (int pass = 2; pass <= iord; pass++) {
    const bool first = (pass == 2), last = (pass == iord);
    if constexpr (sizeof(R) == 8) {
      Q.pairs = P.rho || (P.stdf && !first) ? 1 : 2;
      if (P.stdf && first) LAUNCH(ST_PAIRS, (chain_launch_if(P.chained, k_pairs<R, true, true, true>, grd, blk, 0, s, Q)));
      else if (P.stdf) LAUNCH(ST_PAIRS, (chain_launch_if(P.chained, k_pairs<R, false, false, true>, grd, blk, 0, s, Q)));
      else if (P.rho) LAUNCH(ST_PAIRS, (chain_launch_if(P.chained, k_pairs<R, true, false, false>, grd, blk, 0, s, Q)));
      else if (first) LAUNCH(ST_PAIRS, (chain_launch_if(P.chained, k_pairs<R, true, true, false>, grd, blk, 0, s, Q)));
      else LAUNCH(ST_PAIRS, (chain_launch_if(P.chained, k_pairs<R, false, true, false>, grd, blk, 0, s, Q)));
    }
    if (first) LAUNCH(ST_PSEUDO, (chain_launch_if(P.chained, k_pseudo<R, true>, grd, blk, 0, s, Q)));
    else LAUNCH(ST_PSEUDO, (chain_launch_if(P.chained, k_pseudo<R, false>, grd, blk, 0, s, Q)));
    if (!nonos) LAUNCH(ST_BOUNDS, (chain_launch_if(P.chained, k_bounds<R, false, true, false>, grd, blk, 0, s, P)));
    else if (first && keep) LAUNCH(ST_BOUNDS, (chain_launch_if(P.chained, k_bounds<R, true, true, true>, grd, blk, 0, s, P)));
    else if (first) LAUNCH(ST_BOUNDS, (chain_launch_if(P.chained, k_bounds<R, true, true, false>, grd, blk, 0, s, P)));
    else LAUNCH(ST_BOUNDS, (chain_launch_if(P.chained, k_bounds<R, true, false, true>, grd, blk, 0, s, P)));
    if (nonos) LAUNCH(ST_LIMIT, (chain_launch_if(P.chained, k_limit<R, true>, grd, blk, 0, s, P)));
    else LAUNCH(ST_LIMIT, (chain_launch_if(P.chained, k_limit<R, false>, grd, blk, 0, s, P)));
    if (last) LAUNCH(ST_UPDATE, (chain_launch_if(P.chained, k_update<R, true>, grd, blk, 0, s, P)));
    else LAUNCH(ST_UPDATE, (chain_launch_if(P.chained, k_update<R, false>, grd, blk, 0, s, P)));
  }
  if (P.rho) LAUNCH(ST_RHO_OUT, (chain_launch_if(P.chained, k_rho_out<R, false>, grd, blk, 0, s, P)));
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template int run_step<double>(const Prob<double>&, int, int, Prof*, cudaStream_t);
template int run_step<float>(const Prob<float>&, int, int, Prof*, cudaStream_t);

}  // namespace mpdata
