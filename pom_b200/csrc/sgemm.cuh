// float32 GEMM with FMA instructions (pom_sgemm.cu), as the tensor-core form (pom_gemm_f32.cu) falls back on it.
#pragma once
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace pomk {

// What the split of two operands into planes found out about them (pom_gemm_f32.cu); no words: an unconditional product.
// A word holds, for a part of an operand, the float exponent field of the largest magnitude (254 and up: bf16 cannot
// hold it) above bit 16 and that of the smallest one that is not zero (255: all zeros) below, both of value * 2^24.
struct SgemmFlags {
  const int* a;
  int na;
  const int* b;
  int nb;
  int max_sum;  // largest sum of the two operands' largest exponent fields, smallest sum of their smallest ones,
  int min_sum;  // with which the plane products neither overflow nor lose bits
  struct Range {
    int hi, lo;
  };
  // Of the words first, first + step, ... and the other lanes' (whole warp).
  __device__ __forceinline__ static Range scan(const int* w, int n, int first, int step) {
    int hi = 0, lo = 255;
    for (int i = first; i < n; i += 16 * step) {  // 16 loads in flight (past the end: a word of zeros)
      int v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = i + j * step < n ? __ldcg(w + i + j * step) : 255;
#pragma unroll
      for (int j = 0; j < 16; ++j) hi = max(hi, v[j] >> 16), lo = min(lo, v[j] & 255);
    }
    return Range{__reduce_max_sync(0xffffffffu, hi), __reduce_min_sync(0xffffffffu, lo)};
  }
  __device__ __forceinline__ bool out_of_range(const Range& x, const Range& y) const {
    return x.hi >= 254 || y.hi >= 254 || x.hi + y.hi > max_sum || x.lo + y.lo < min_sum;
  }
  // Whether the planes cannot carry the product.
  __device__ __forceinline__ bool any_in_warp(int lane) const {
    return out_of_range(scan(a, na, lane, 32), scan(b, nb, lane, 32));
  }
  __device__ __forceinline__ bool any_in_block() const {
    __shared__ int4 sh[8];  // per warp (blocks of up to 256 threads)
    Range x = scan(a, na, threadIdx.x, blockDim.x), y = scan(b, nb, threadIdx.x, blockDim.x);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_int4(x.hi, x.lo, y.hi, y.lo);
    __syncthreads();
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
      const int4 v = sh[w];
      x = Range{max(x.hi, v.x), min(x.lo, v.y)}, y = Range{max(y.hi, v.z), min(y.lo, v.w)};
    }
    return out_of_range(x, y);
  }
};

}  // namespace pomk

namespace pomh {
// C (+)= alpha * A·Bᵀ (pom_sgemm.cu).  With flag words: only if one of them is up.
int launch_sgemm(const pom_gemm_args* a, const pomk::SgemmFlags& flags, cudaStream_t st);
}  // namespace pomh
