// float32 GEMM with FMA instructions (pom_sgemm.cu), as the tensor-core form (pom_gemm_f32.cu) falls back on it.
#pragma once
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace pomk {

// Marks that the split of two operands into planes left behind (pom_gemm_f32.cu); no words: an unconditional product.
struct SgemmFlags {
  const int* a;
  int na;
  const int* b;
  int nb;
  __device__ __forceinline__ bool scan(int first, int step) const {
    int f = 0;
    for (int i = first; i < na; i += step) f |= __ldcg(a + i);
    for (int i = first; i < nb; i += step) f |= __ldcg(b + i);
    return f != 0;
  }
  __device__ __forceinline__ bool any_in_warp(int lane) const { return __any_sync(0xffffffffu, scan(lane, 32)); }
  __device__ __forceinline__ bool any_in_block() const { return __syncthreads_or(scan(threadIdx.x, blockDim.x)); }
};

}  // namespace pomk

namespace pomh {
// C (+)= alpha * A·Bᵀ (pom_sgemm.cu).  With flag words: only if one of them is up.
int launch_sgemm(const pom_gemm_args* a, const pomk::SgemmFlags& flags, cudaStream_t st);
}  // namespace pomh
