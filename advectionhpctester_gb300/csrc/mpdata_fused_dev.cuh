// Helpers that the fused single-precision kernels share (mpdata_fused.cu,
// mpdata_narrow.cu): staging by TMA and cp.async, bounded mbarrier waits,
// NaN-propagating extrema, work items, the arena's tensor map.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mpdata_fused.cuh"

namespace mpdata {
namespace {

__device__ __forceinline__ int wrapn(int i, int n) {
  int r = (i - 1) % n;
  if (r < 0) r += n;
  return r + 1;
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint64_t* m, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* m, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* m, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(m)), "r"(parity), "r"(1000000u)
      : "memory");
  return ok != 0;
}
// Bounded wait on an mbarrier phase: false when the limit ran out.  Each
// try_wait suspends the thread until the phase completes or about 1 ms has
// passed, so a waiting warp issues almost nothing and the limit is seconds.
__device__ __forceinline__ bool mbar_wait(uint64_t* m, uint32_t parity) {
  for (int it = 0; it < 4096; it++)
    if (mbar_try_wait(m, parity)) return true;
  return false;
}
// One box of arena field f, plane z (0-based), into dst.  x must be a
// multiple of 4 (16 bytes of FP32).
__device__ __forceinline__ void tma_box(float* dst, const CUtensorMap* map, int x, int y, int z, int f,
                                        uint64_t* m) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(f), "r"(smem_u32(m))
      : "memory");
}

// Dynamic shared memory rounded up to 128 bytes, the alignment a TMA box
// destination needs (every staged plane is a multiple of 128 bytes from it).
__device__ __forceinline__ float* smem_base() {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t off = smem_u32(smem_raw);
  return reinterpret_cast<float*>(smem_raw + ((128u - (off & 127u)) & 127u));
}

typedef FusedArgs FzArgs;

// The fields of one pass: which arena fields hold its input field, its
// output field and the running extrema it reads and writes (the same for
// every problem of a batch).
struct FzPass {
  int fin, fout, fmx_in, fmn_in, fmx_out, fmn_out;
  __device__ __forceinline__ void apply(FzArgs& a) const {
    a.fin = fin;
    a.fout = fout;
    a.fmx_in = fmx_in;
    a.fmn_in = fmn_in;
    a.fmx_out = fmx_out;
    a.fmn_out = fmn_out;
  }
};

__device__ __forceinline__ int mod3(int a) { return a >= 3 ? a - 3 : a; }  // a in [0, 5]
__device__ __forceinline__ bool is1(float v) { return __float_as_int(v) == 0x3f800000; }

// NaN-propagating max and min (one instruction each).
__device__ __forceinline__ float maxn(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float minn(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// One work item of a batch.
struct Item {
  int p, bxi, byi, bzi;
};
__device__ __forceinline__ Item item_of(const unsigned long long* items) {
  const unsigned long long w = items[blockIdx.x];
  return Item{(int)(w & 0xffffu), (int)((w >> 16) & 0xffffu), (int)((w >> 32) & 0xffffu), (int)(w >> 48)};
}

template <class K>
int set_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess ? 0
                                                                                                                : -5;
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The tensor map of an arena: rows of px floats, planes of so many rows, lp
// planes a field, and a box of bx x by cells of one plane.  0 on success.
int encode_arena(CUtensorMap* map, float* arena, int px, int rows, int lp, int fields, int bx, int by) {
  static EncodeTiled enc = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<EncodeTiled>(fn);
  }();
  if (!enc) return -5;
  const cuuint64_t row = (cuuint64_t)px * 4, plane = row * rows;
  const cuuint64_t dims[4] = {(cuuint64_t)px, (cuuint64_t)rows, (cuuint64_t)lp, (cuuint64_t)fields};
  const cuuint64_t strides[3] = {row, plane, plane * lp};
  const cuuint32_t box[4] = {(cuuint32_t)bx, (cuuint32_t)by, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, arena, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -5;
}

// the arena fields of the next pass: it reads this pass's output field and extrema
static void next_pass(int& fin, int& fout, int& mxi, int& mni, int& mxo, int& mno) {
  fin = fout;
  fout = fout == FZ_X1 ? FZ_X0 : FZ_X1;
  mxi = mxo;
  mni = mno;
  mxo = mxo == FZ_MX0 ? FZ_MX1 : FZ_MX0;
  mno = mno == FZ_MN0 ? FZ_MN1 : FZ_MN0;
}

#define FZ_LAUNCH(stage, ...)              \
  do {                                     \
    if (prof) prof->begin(stage, s);       \
    __VA_ARGS__;                           \
    if (prof) prof->end(stage, s);         \
    add_launches(1);                       \
  } while (0)

}  // namespace
}  // namespace mpdata
