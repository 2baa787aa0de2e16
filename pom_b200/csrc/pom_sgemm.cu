// float32 GEMM with FMA instructions: every output is one chain of fused multiply-adds over k = 0, 1, 2, ... from zero.
//
// The order does not depend on the tile, the batch or the operands' storage order.  Products with a short K, and those
// that the three-plane form (pom_gemm_f32.cu) cannot carry, come here.
//
// What bounds it: FMA issue (74 TFLOP/s at 1.965 GHz; 48 reached at 4080 x 4608 x 1152, where 4 x 4 outputs per thread
// and a single buffer reach 22, 8 x 16 outputs at one block per SM 47, scalar FMAs 44).  A thread keeps TM x 8 outputs, so
// that 4 (or 3) shared-memory reads feed 64 (or 32) FMAs; the next k-step is loaded into registers while the current one is computed from a
// double-buffered tile, one barrier per step.
#include "common.cuh"
#include "sgemm.cuh"

using namespace pomk;
using namespace pomh;

namespace {

constexpr int kStep = 16;  // k elements per step

struct SgemmOperand {
  const float* p;
  long long ld;
  int rows;  // extent of the M or N dimension
  int mn;    // 1: stored (K, rows), 0: stored (rows, K)
  int vec;   // 16-byte loads are possible (base and leading dimension)
};

// This thread's share of a TILE x kStep block: TILE * kStep / NT values in 16-byte pieces.  K-major: four lanes take the
// 64 bytes of a row and store them transposed (rows of TILE + 4 floats: two-way bank conflicts); MN-major: pieces of a
// k-row.
template <int TILE, int NT>
struct BlockLoader {
  static constexpr int kValues = TILE * kStep / NT;  // 4 or 8
  static constexpr int kPieces = kValues / 4;
  float4 v[kPieces];

  __device__ __forceinline__ void load(const SgemmOperand& o, int row0, int k0, int K, int tid) {
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {
      int r, k;
      if (!o.mn) {
        r = tid / 4 + j * (NT / 4), k = (tid % 4) * 4;
      } else {
        const int piece = tid + j * NT;
        r = (piece % (TILE / 4)) * 4, k = piece / (TILE / 4);
      }
      const int gr = row0 + r, gk = k0 + k;
      const float* s = o.p + (o.mn ? gk * o.ld + gr : gr * o.ld + gk);
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      const bool outer = o.mn ? gk < K : gr < o.rows;
      const int left = o.mn ? o.rows - gr : K - gk;
      if (outer) {
        if (o.vec && left >= 4) {
          x = __ldg(reinterpret_cast<const float4*>(s));
        } else {
          if (left > 0) x.x = __ldg(s);
          if (left > 1) x.y = __ldg(s + 1);
          if (left > 2) x.z = __ldg(s + 2);
          if (left > 3) x.w = __ldg(s + 3);
        }
      }
      v[j] = x;
    }
  }
  __device__ __forceinline__ void store(float (*s)[TILE + 4], int mn, int tid) const {
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {
      if (!mn) {
        const int r = tid / 4 + j * (NT / 4), k = (tid % 4) * 4;
        s[k][r] = v[j].x, s[k + 1][r] = v[j].y, s[k + 2][r] = v[j].z, s[k + 3][r] = v[j].w;
      } else {
        const int piece = tid + j * NT;
        *reinterpret_cast<float4*>(&s[piece / (TILE / 4)][(piece % (TILE / 4)) * 4]) = v[j];
      }
    }
  }
};

__device__ __forceinline__ void fma2(float2& d, float a, float2 b) {
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 z, {%0, %1};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}"
      : "+f"(d.x), "+f"(d.y)
      : "f"(a), "f"(b.x), "f"(b.y));
}

// TILE x TILE outputs by NT threads, TM rows x 8 columns each.
template <int TILE, int NT, int TM>
__global__ void __launch_bounds__(NT, TILE == 128 ? 2 : 4)
sgemm_kernel(const SgemmOperand A, const SgemmOperand Bm, float* __restrict__ C, int K, long long ldc, float alpha,
             int accumulate, const SgemmFlags flags) {
  constexpr int kCols = TILE / 8;  // threads along n
  static_assert(NT == kCols * (TILE / TM), "thread layout");
  __shared__ __align__(16) float As[2][kStep][TILE + 4];
  __shared__ __align__(16) float Bs[2][kStep][TILE + 4];
  const int tid = threadIdx.x, tx = tid % kCols, ty = tid / kCols;
  griddep_wait();
  griddep_launch();
  if (flags.na + flags.nb > 0 && !flags.any_in_block()) return;
  const int M = A.rows, N = Bm.rows;
  const int tiles_n = (N + TILE - 1) / TILE;
  const long long tiles = 1ll * tiles_n * ((M + TILE - 1) / TILE);
  const int steps = (K + kStep - 1) / kStep;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int m0 = static_cast<int>(tile / tiles_n) * TILE, n0 = static_cast<int>(tile % tiles_n) * TILE;
    BlockLoader<TILE, NT> la, lb;
    la.load(A, m0, 0, K, tid);
    lb.load(Bm, n0, 0, K, tid);
    float2 acc[TM][4] = {};
    la.store(As[0], A.mn, tid);
    lb.store(Bs[0], Bm.mn, tid);
    __syncthreads();
    for (int st = 0; st < steps; ++st) {
      const int cur = st & 1;
      if (st + 1 < steps) {
        la.load(A, m0, (st + 1) * kStep, K, tid);
        lb.load(Bm, n0, (st + 1) * kStep, K, tid);
      }
#pragma unroll
      for (int k = 0; k < kStep; ++k) {
        float a[TM];
        float2 b[4];
        // a thread's rows and columns lie in groups of four, so that a warp's reads of one instruction are adjacent
#pragma unroll
        for (int i = 0; i < TM; i += 4)
          *reinterpret_cast<float4*>(a + i) =
              *reinterpret_cast<const float4*>(&As[cur][k][(i / 4) * (TILE * 4 / TM) + ty * 4]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float4 q = *reinterpret_cast<const float4*>(&Bs[cur][k][j * (TILE / 2) + tx * 4]);
          b[2 * j] = make_float2(q.x, q.y), b[2 * j + 1] = make_float2(q.z, q.w);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) fma2(acc[i][j], a[i], b[j]);
      }
      if (st + 1 < steps) {
        la.store(As[cur ^ 1], A.mn, tid);
        lb.store(Bs[cur ^ 1], Bm.mn, tid);
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + (i / 4) * (TILE * 4 / TM) + ty * 4 + (i & 3);
      if (gm >= M) continue;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int gn = n0 + j * (TILE / 2) + tx * 4;
        const float o[4] = {alpha * acc[i][2 * j].x, alpha * acc[i][2 * j].y, alpha * acc[i][2 * j + 1].x,
                            alpha * acc[i][2 * j + 1].y};
        float* c = C + static_cast<long long>(gm) * ldc + gn;
        if (gn + 4 <= N && !accumulate && (reinterpret_cast<uintptr_t>(c) & 15) == 0) {
          *reinterpret_cast<float4*>(c) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (gn + e < N) c[e] = accumulate ? c[e] + o[e] : o[e];
        }
      }
    }
  }
}

template <int TILE, int NT, int TM>
cudaError_t start(const SgemmOperand& A, const SgemmOperand& Bm, const pom_gemm_args* a, const SgemmFlags& flags,
                  cudaStream_t st) {
  const long long tiles = ceil_div(A.rows, TILE) * ceil_div(Bm.rows, TILE);
  // behind a tensor-core product this is the exception: few blocks, which walk the tiles if they have to
  const long long cap = flags.na + flags.nb > 0 ? 2ll * sm_count() : INT32_MAX;
  return launch_pdl(sgemm_kernel<TILE, NT, TM>, dim3(static_cast<unsigned>(tiles < cap ? tiles : cap)), dim3(NT), 0, st,
                    A, Bm, static_cast<float*>(a->C), static_cast<int>(a->K), static_cast<long long>(a->ldc), a->alpha,
                    static_cast<int>(a->out_mode == POM_OUT_F32_ACCUM), flags);
}

}  // namespace

namespace pomh {

int launch_sgemm(const pom_gemm_args* a, const SgemmFlags& flags, cudaStream_t st) {
  const auto operand = [](const void* p, int64_t ld, int64_t rows, int mn) {
    return SgemmOperand{static_cast<const float*>(p), ld, static_cast<int>(rows), mn, aligned16(p) && ld % 4 == 0};
  };
  const SgemmOperand A = operand(a->A, a->lda, a->M * a->batches, a->a_mn_major != 0);
  const SgemmOperand B = operand(a->Bm, a->ldb, a->N, a->b_mn_major != 0);
  // 64-wide tiles spread a small product over four times as many SMs; they read a third more shared memory per FMA
  const double wide = static_cast<double>(ceil_div(ceil_div(A.rows, 128) * ceil_div(B.rows, 128), sm_count())) * 4.0;
  const double narrow = static_cast<double>(ceil_div(ceil_div(A.rows, 64) * ceil_div(B.rows, 64), sm_count())) * 1.25;
  if ((narrow < wide ? start<64, 128, 4>(A, B, a, flags, st) : start<128, 256, 8>(A, B, a, flags, st)) != cudaSuccess) {
    (void)cudaGetLastError();
    return POM_ERR_CUDA;
  }
  count_launch();
  return check_launch();
}

}  // namespace pomh

extern "C" int pom_gemm_f32(const pom_gemm_args* a, void* stream) {
  if (!a || !a->A || !a->Bm || !a->C) return POM_ERR_NULL;
  if (a->M <= 0 || a->N <= 0 || a->K <= 0 || a->batches <= 0) return POM_ERR_BAD_SHAPE;
  if (a->out_mode != POM_OUT_F32 && a->out_mode != POM_OUT_F32_ACCUM) return POM_ERR_UNSUPPORTED;
  if (a->a_mn_major && a->batches != 1) return POM_ERR_UNSUPPORTED;
  const long long Mtot = a->M * a->batches;
  if (Mtot > INT32_MAX || a->N > INT32_MAX || a->K > INT32_MAX) return POM_ERR_TOO_LARGE;
  if (ceil_div(Mtot, 64) > 65535) return POM_ERR_TOO_LARGE;
  return launch_sgemm(a, SgemmFlags{nullptr, 0, nullptr, 0, 0, 0}, static_cast<cudaStream_t>(stream));
}
