// Counts where the FP32 quotients of mpdata_quot32.cuh differ from IEEE division
// (one thread an operand, counters by atomics; every operand is made here).
#include <cuda_runtime.h>
#include <stdint.h>

#include "mpdata_quot32.cuh"

namespace {

__device__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  return x ^ (x >> 16);
}
__device__ float make(uint32_t sign, int e, uint32_t significand) {  // exponent e, 23 fraction bits
  return __uint_as_float(sign << 31 | (uint32_t)(e + 127) << 23 | (significand & 0x7fffffu));
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// count[0]: wrong, count[1]: taken by the fast path
__device__ void check(float n, float d, unsigned long long* count) {
  bool slow = false;
  const float q = mpdata::quot_fast(n, d, slow);
  if (slow) return;
  atomicAdd(count + 1, 1ULL);
  if (!same(q, n / d)) atomicAdd(count, 1ULL);
}

// every significand at exponent e: 1/d
__global__ void reciprocals(int e, unsigned long long* count) {
  const float d = make(0, e, blockIdx.x * blockDim.x + threadIdx.x);
  if (mpdata::den_slow(d)) return;
  atomicAdd(count + 1, 1ULL);
  if (!same(mpdata::rcp_fast(d), 1.0f / d)) atomicAdd(count, 1ULL);
}

// every odd significand D of the divisor with a numerator N such that N*2^25 = D*Q + r,
// Q odd: the quotient is a middle of two numbers and r/D of a unit beside it
__global__ void middles(int r, int ed, int eq, unsigned long long* count) {
  const uint32_t D = (blockIdx.x * blockDim.x + threadIdx.x) * 2 + 1 + (1u << 23);
  uint32_t inv = D;  // D*D = 1 mod 8: three bits, doubled by each step
  for (int s = 0; s < 4; s++) inv *= 2 - D * inv;
  const uint32_t Q = (0u - (uint32_t)r * inv) & 0x1ffffffu;  // 25 bits
  if (Q < 1u << 24) return;
  const uint64_t N = ((uint64_t)D * Q + (int64_t)r) >> 25;
  if (N < 1u << 23 || N >= 1u << 24) return;
  const float d = make(0, ed, D), n = make(D >> 1 & 1, 0, (uint32_t)N);
  check(ldexpf(n, ed + eq), d, count);
}

// random operands: n of exponents n0..n1 (subnormals below -126), d of d0..d1
__global__ void randoms(uint32_t seed, int n0, int n1, int d0, int d1, unsigned long long* count) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t a = hash32(t * 4 + seed), b = hash32(t * 4 + 1 + seed), c = hash32(t * 4 + 2 + seed);
  const int en = n0 + (int)((c & 0xffffu) % (uint32_t)(n1 - n0 + 1));
  const int ed = d0 + (int)((c >> 16) % (uint32_t)(d1 - d0 + 1));
  const float d = make(0, ed, b);
  const float n = en >= -126 ? make(a >> 31, en, a)
                             : __uint_as_float((a & 0x80000000u) | ((a & 0x7fffffu) | 0x800000u) >> (-126 - en));
  check(n, d, count);
}

int result(unsigned long long* dev, unsigned long long* host) {
  const cudaError_t e = cudaMemcpy(host, dev, 2 * sizeof(*dev), cudaMemcpyDeviceToHost);
  const cudaError_t f = cudaFree(dev);
  return e == cudaSuccess && f == cudaSuccess ? 0 : -1;
}
unsigned long long* counters() {
  unsigned long long* p = nullptr;
  if (cudaMalloc(&p, 2 * sizeof(*p)) != cudaSuccess || cudaMemset(p, 0, 2 * sizeof(*p)) != cudaSuccess) return nullptr;
  return p;
}

}  // namespace

extern "C" int check_reciprocals(int e, unsigned long long* out) {
  unsigned long long* c = counters();
  if (!c) return -1;
  reciprocals<<<(1 << 23) / 256, 256>>>(e, c);
  return result(c, out);
}
extern "C" int check_middles(int r, int ed, int eq, unsigned long long* out) {
  unsigned long long* c = counters();
  if (!c) return -1;
  middles<<<(1 << 22) / 256, 256>>>(r, ed, eq, c);
  return result(c, out);
}
extern "C" int check_randoms(unsigned seed, int n0, int n1, int d0, int d1, unsigned long long* out) {
  unsigned long long* c = counters();
  if (!c) return -1;
  randoms<<<(1 << 26) / 256, 256>>>(seed, n0, n1, d0, d1, c);
  return result(c, out);
}
