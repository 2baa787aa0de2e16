// float32 GEMM on the tensor cores: C[m, n] = alpha * sum_k A[m, k] * B[n, k] with the accuracy of float32 sums.
//
// Every float32 operand is first written as three bf16 planes of 2^24 x (round to nearest, then the remainders), which
// hold all 24 bits of it: 2^24 x = hi + mid + lo, |mid| <= 2^-9 |hi|, |lo| <= 2^-18 |hi| (without the factor the last
// bits of |x| < 2^-110 would fall under bf16's range).  Of the nine plane products the six largest are formed (hi·hi,
// hi·mid, mid·hi, mid·mid, hi·lo, lo·hi); the three left out are below 2^-26 of the product.  The sum times 2^-48 is the
// result.
// A long sum in a tensor-memory accumulator is taken to lose up to a unit in its last place per instruction (how tcgen05
// rounds is not documented).  Two measures keep the result at least as close to the exact sum as a chain of float32 FMAs:
//   * hi·hi is summed in tensor memory over one 64-deep k-block only (four instructions); the epilogue warps add each
//     block into registers with correctly rounded float32 additions while the next products run;
//   * the five small products go into an accumulator of their own, whose losses are 2^-8 of the other's.
//
// What bounds it: the tensor pipe, six bf16 products per float32 product (229 TFLOP/s of float32 work at this card's
// sustained bf16 rate; 4080 x 4608 x 1152 takes 193 us = 224 TFLOP/s, 1969 us with FMAs; error against 64 bits 1.1e-7,
// 6.1e-7 with FMAs).  A pair tile of 256 x 256 loads 96 KB per SM and k-block for 3072 tensor cycles (32 B/clk/SM,
// half of what the bf16 kernels ask of L2), so two stages of three planes are enough.
//
// Operands whose products could leave the range in which all of this holds do not go through the planes.  The split notes
// the exponents of the largest and the smallest magnitude (but zero) of either operand.  The largest product times K has to
// stay below 2^78 (2^126 with the factors: no sum overflows), the smallest at or above 2^-148 (2^-100 with the factors:
// no plane product that counts falls under 2^-126, where a tensor core may take it for zero).  Otherwise, and for
// infinities and NaN, the FMA kernel (sgemm_kernel) computes the product, decided on the device without the host.
#include <cfloat>
#include <cmath>
#include <cudaTypedefs.h>
#include "common.cuh"
#include "gemm_launch.cuh"
#include "sgemm.cuh"

using namespace pomk;
using namespace pomh;

namespace {

constexpr int kFlagWords = 1024;                // one word per block of the split kernel
constexpr int kFlagBytes = kFlagWords * 4;
constexpr int kSplitThreads = 256;
constexpr int kF32Threads = 32 * 10;            // producer, MMA issuer, eight epilogue warps
constexpr float kScale = 0x1p24f, kUnscale = 0x1p-48f;  // of an operand's planes, of a product of two
constexpr int kMinSplitBlocks = 2;              // k-blocks that a K split keeps at least

inline int64_t plane_ld(int64_t cols) { return (cols + 7) / 8 * 8; }
// Blocks of either split kernel, and words in the buffer: a function of the operand alone, so that planes filled by one
// call are read rightly by another.
inline int split_blocks(int64_t rows, int64_t cols) {
  const int64_t n = ceil_div(rows * (plane_ld(cols) / 8), kSplitThreads);
  return static_cast<int>(n < kFlagWords ? n : kFlagWords);
}
inline __nv_bfloat16* planes_of(void* buf) {
  return reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(buf) + kFlagBytes);
}

// ---------------------------------------------------------------------------- split into planes
struct SplitMat {
  const float* src;
  uint4* dst;       // three planes of rows x ldp bf16
  int* flags;       // word of every block: exponents of its largest and smallest magnitudes (SgemmFlags)
  long long rows, cols, ld, groups;  // groups of 8 columns per row
  int blocks;
};

// Eight values of a row, zero past its end.
__device__ __forceinline__ void load8(const float* s, long long left, bool vec, float (&v)[8]) {
  if (vec && left >= 8) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(s)), y = __ldg(reinterpret_cast<const float4*>(s) + 1);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w, v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = e < left ? __ldg(s + e) : 0.f;
  }
}

// Largest and smallest magnitude (but zero) of the values a thread splits, as bits.
struct Extremes {
  uint32_t hi = 0, lo = 0xffffffffu;  // lo: less one, so that zero comes out on top
  __device__ __forceinline__ void see(float x) {
    const uint32_t u = __float_as_uint(x) & 0x7fffffffu;
    hi = max(hi, u);
    lo = min(lo, u - 1u);
  }
  __device__ __forceinline__ void add(const Extremes& o) { hi = max(hi, o.hi), lo = min(lo, o.lo); }
  // The word of the block (every thread calls it once).
  __device__ __forceinline__ void store(int* word) const {
    __shared__ uint32_t sh[2][kSplitThreads / 32];
    const uint32_t h = __reduce_max_sync(0xffffffffu, hi), l = __reduce_min_sync(0xffffffffu, lo);
    if ((threadIdx.x & 31) == 0) sh[0][threadIdx.x >> 5] = h, sh[1][threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t a = sh[0][0], b = sh[1][0];
      for (int w = 1; w < kSplitThreads / 32; ++w) a = max(a, sh[0][w]), b = min(b, sh[1][w]);
      *word = static_cast<int>(a >> 23 << 16 | (b == 0xffffffffu ? 255u : (b + 1u) >> 23));
    }
  }
};

// Planes of 2^24 a and 2^24 b.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t (&o)[3], Extremes& x) {
  a *= kScale, b *= kScale;
  x.see(a), x.see(b);
  o[0] = pack_bf16x2(a, b);
  a -= __uint_as_float(o[0] << 16), b -= __uint_as_float(o[0] & 0xffff0000u);
  o[1] = pack_bf16x2(a, b);
  a -= __uint_as_float(o[1] << 16), b -= __uint_as_float(o[1] & 0xffff0000u);
  o[2] = pack_bf16x2(a, b);
}

// Memory-bound (4 bytes read, 6 written per value); blockIdx.y picks the operand, so that both operands of a small
// product are one launch.
__global__ void __launch_bounds__(kSplitThreads) split_planes_kernel(const SplitMat m0, const SplitMat m1) {
  griddep_wait();
  griddep_launch();
  const SplitMat& m = blockIdx.y ? m1 : m0;
  if (static_cast<int>(blockIdx.x) >= m.blocks) return;
  const long long total = m.rows * m.groups, plane = total;
  const bool vec = (m.ld & 3) == 0 && (reinterpret_cast<uintptr_t>(m.src) & 15) == 0;
  Extremes seen;
  for (long long i = blockIdx.x * 1ll * kSplitThreads + threadIdx.x; i < total; i += 1ll * m.blocks * kSplitThreads) {
    const long long r = i / m.groups, c = (i - r * m.groups) * 8;
    float v[8];
    load8(m.src + r * m.ld + c, m.cols - c, vec, v);
    uint32_t p[4][3];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      split_pair(v[2 * e], v[2 * e + 1], p[e], seen);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) m.dst[k * plane + i] = make_uint4(p[0][k], p[1][k], p[2][k], p[3][k]);
  }
  seen.store(m.flags + blockIdx.x);
}

// The same with a warp per row, which also leaves the row's 2-norm (pom_project_f32): 0 only for a row of zeros, and never
// too small where squares underflow (sqrt(cols) times the largest magnitude then).
__global__ void __launch_bounds__(kSplitThreads) split_rows_kernel(const SplitMat m0, const SplitMat m1,
                                                                   float* __restrict__ norms) {
  griddep_wait();
  griddep_launch();
  const SplitMat& m = blockIdx.y ? m1 : m0;
  if (static_cast<int>(blockIdx.x) >= m.blocks) return;
  float* norm = norms + (blockIdx.y ? m0.rows : 0);
  const int lane = threadIdx.x & 31, warps = kSplitThreads / 32;
  const bool vec = (m.ld & 3) == 0 && (reinterpret_cast<uintptr_t>(m.src) & 15) == 0;
  const long long plane = m.rows * m.groups;
  Extremes seen;
  for (long long r = blockIdx.x * 1ll * warps + (threadIdx.x >> 5); r < m.rows; r += 1ll * m.blocks * warps) {
    float sq = 0.f;
    Extremes row;
    for (long long g = lane; g < m.groups; g += 32) {
      float v[8];
      load8(m.src + r * m.ld + g * 8, m.cols - g * 8, vec, v);
      uint32_t p[4][3];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sq = fmaf(v[2 * e], v[2 * e], fmaf(v[2 * e + 1], v[2 * e + 1], sq));
        split_pair(v[2 * e], v[2 * e + 1], p[e], row);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        m.dst[k * plane + r * m.groups + g] = make_uint4(p[0][k], p[1][k], p[2][k], p[3][k]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    seen.add(row);
    const float top = __uint_as_float(__reduce_max_sync(0xffffffffu, row.hi)) * (1.f / kScale);
    if (lane == 0) norm[r] = sq < 0x1p-60f ? top * sqrtf(static_cast<float>(m.cols)) : sqrtf(sq);
  }
  seen.store(m.flags + blockIdx.x);
}

// ---------------------------------------------------------------------------- chain values beside the kinks
struct NearArgs {
  const float* A;
  const float* B;
  float* C;
  const float* norms;  // 2-norms of the M rows of A, then of the N rows of B
  const float* bias;   // of the gate columns
  long long lda, ldb, ldc;
  int M, N, K;
  int gate0;           // columns from here on are gate columns
  float factor;
};

// C = A·Bᵀ as the planes gave it -> elements so close to a kink (activation: 0, 6, -10; gate: -3 and 3 after its bias)
// that the FMA chain's rounding could put them on the other side get the chain's own value, bit for bit that of
// sgemm_kernel.  Both sums are within factor * |a| |b| of one another, factor = 8 sqrt(K) 2^-24: a chain's error stays
// below lambda sqrt(K) 2^-24 sum |a_k b_k| but for a probability of 2 exp(-lambda^2 / 2) (Higham and Mary, 2019; 8: 3e-14),
// the planes' is a fifth of it, and sum |a_k b_k| <= |a| |b|.  Of dense inputs one element in about 3000 is that close.
// Where a row of A or of B is all zeros (a padded token) both sums are exactly 0 and there is no chain to run.
// The float32 training step at 4 x 1020 x 1152 takes 1429 us with this and 1952 with the FMA chain for every element.
__global__ void __launch_bounds__(256) near_kinks_kernel(const NearArgs a) {
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31;
  const int per_row = (a.N + 3) / 4;
  const long long total = 1ll * a.M * per_row, stride = gridDim.x * 256ll;
  for (long long base = blockIdx.x * 256ll + (threadIdx.x - lane); base < total; base += stride) {
    const long long i = base + lane;
    const bool on = i < total;
    const long long r = on ? i / per_row : 0;
    const int c0 = on ? static_cast<int>(i - r * per_row) * 4 : 0;
    float* row = a.C + r * a.ldc + c0;
    float v[4];
    if (c0 + 4 <= a.N && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
      const float4 q = *reinterpret_cast<const float4*>(row);
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = c0 + e < a.N ? row[e] : 0.f;
    }
    const float na = __ldg(a.norms + r);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = min(c0 + e, a.N - 1);
      const float nb = __ldg(a.norms + a.M + c), eps = fmaxf(a.factor * (na * nb), FLT_MIN);
      const bool gate = c >= a.gate0;
      const float x = gate ? fabsf(v[e] + __ldg(a.bias + c - a.gate0)) : v[e];
      const bool near = gate ? fabsf(x - 3.f) <= eps
                             : fabsf(x) <= eps || fabsf(x - 6.f) <= eps || fabsf(x + 10.f) <= eps;
      // (a sum that is not finite has come from the FMA kernel already)
      uint32_t todo = __ballot_sync(0xffffffffu, on && c0 + e < a.N && near && eps < FLT_MAX && na > 0.f && nb > 0.f);
      while (todo) {  // the whole warp brings the element's two rows, 128 k ahead; every lane runs the chain
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const float* pa = a.A + __shfl_sync(0xffffffffu, r, src) * a.lda;
        const float* pb = a.B + static_cast<long long>(__shfl_sync(0xffffffffu, c, src)) * a.ldb;
        float acc = 0.f, xa[4], xb[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int k = 32 * q + lane;
          xa[q] = k < a.K ? __ldg(pa + k) : 0.f, xb[q] = k < a.K ? __ldg(pb + k) : 0.f;
        }
        for (int k0 = 0; k0 < a.K; k0 += 128) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float ca = xa[q], cb = xb[q];
            const int k = k0 + 128 + 32 * q + lane, left = a.K - k0 - 32 * q;
            xa[q] = k < a.K ? __ldg(pa + k) : 0.f, xb[q] = k < a.K ? __ldg(pb + k) : 0.f;
            if (left >= 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                acc = fmaf(__shfl_sync(0xffffffffu, ca, j), __shfl_sync(0xffffffffu, cb, j), acc);
            } else {
              for (int j = 0; j < left; ++j)
                acc = fmaf(__shfl_sync(0xffffffffu, ca, j), __shfl_sync(0xffffffffu, cb, j), acc);
            }
          }
        }
        if (lane == src) row[e] = acc;
      }
    }
  }
}

// ---------------------------------------------------------------------------- the GEMM
struct F32Out {
  float* C;
  long long ldc, split_stride;  // split_stride > 0: every K split stores its partial sums at C + split * stride
  float alpha;   // times kUnscale
  int accumulate;
  SgemmFlags flags;
};

template <int BN>
struct F32Cfg {
  static constexpr int kHalfN = BN / 2;
  static constexpr int kAPlane = kBM * kBK * 2;
  static constexpr int kBPlane = kHalfN * kBK * 2;
  static constexpr int kStageBytes = 3 * (kAPlane + kBPlane);
  static constexpr int kStages = BN == 256 ? 2 : 3;
  static constexpr int kMainBufs = BN == 256 ? 1 : 2;  // 512 tensor-memory columns: [main x bufs][small x bufs]
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
};

// One 256 x BN output tile per cluster of two CTAs (gemm2_sm100.cuh has the pair protocol).  Per k-block the issuer
// runs hi·hi into a main accumulator, then the five small products; the epilogue drains the main accumulator during
// the latter, so one main buffer is enough at BN = 256.
template <int BN, bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kF32Threads, 1)
gemm_f32_planes_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const GemmGeom geom, const F32Out out, int* __restrict__ status) {
  using Cfg = F32Cfg<BN>;
  constexpr int ST = Cfg::kStages, MB = Cfg::kMainBufs;
  constexpr uint32_t kIdesc = make_idesc_bf16_m256(BN, A_MN, B_MN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + ST * Cfg::kStageBytes);
  uint64_t* full_bar = bars;            // leader: planes of a stage have landed in both CTAs
  uint64_t* empty_bar = bars + ST;      // both CTAs
  uint64_t* mfull = bars + 2 * ST;      // both CTAs: hi·hi of a k-block is complete
  uint64_t* mempty = mfull + MB;        // leader: ... and has been added into registers by both CTAs
  uint64_t* cfull = mempty + MB;        // the same pair for the small products of a tile
  uint64_t* cempty = cfull + MB;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(cempty + MB);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) mbar_init(&full_bar[s], 1), mbar_init(&empty_bar[s], 1);
    for (int a = 0; a < MB; ++a) {
      mbar_init(&mfull[a], 1), mbar_init(&cfull[a], 1);
      mbar_init(&mempty[a], 2 * kEpiWarps), mbar_init(&cempty[a], 2 * kEpiWarps);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc2(tmem_holder, 512);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t tmem_small = tmem_base + MB * BN;
  griddep_wait();
  griddep_launch();

  const int total_units = pairs_of(geom) * geom.n_tiles * geom.split_k;
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs): three planes per load
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      for (int unit = cluster_id; unit < total_units && alive; unit += n_clusters) {
        const TileCtx t = decode_pair_tile(geom, unit, BN, rank);
        const int kb0 = t.split * geom.kb_per_split, kb1 = min(geom.k_blocks, kb0 + geom.kb_per_split);
        const int bcol = t.col0 + static_cast<int>(rank) * Cfg::kHalfN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, status, kStatusProducerTimeout)) {
            alive = false;
            break;
          }
          uint8_t* sa = tiles + stage * Cfg::kStageBytes;
          uint8_t* sb = sa + 3 * Cfg::kAPlane;
          const uint32_t full0 = map_to_cta(smem_u32(&full_bar[stage]), 0);
          if (leader) mbar_expect_tx(&full_bar[stage], 2 * Cfg::kStageBytes);
          if constexpr (!A_MN) {
            tma2_load_3d(sa, &tmA, full0, kb * kBK, t.row0, 0);
          } else {
#pragma unroll
            for (int j = 0; j < kBM / 64; ++j)
              tma2_load_3d(sa + j * 3 * (kBK * 128), &tmA, full0, t.row0 + j * 64, kb * kBK, 0);
          }
          if constexpr (!B_MN) {
            tma2_load_3d(sb, &tmB, full0, kb * kBK, bcol, 0);
          } else {
#pragma unroll
            for (int j = 0; j < Cfg::kHalfN / 64; ++j)
              tma2_load_3d(sb + j * 3 * (kBK * 128), &tmB, full0, bcol + j * 64, kb * kBK, 0);
          }
          if (++stage == ST) stage = 0, phase ^= 1u;
        }
      }
      if (!alive)
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (leader && lane == 0) {
      // Plane p of a stage.  K-major: whole planes follow one another; MN-major: the planes of a 64-wide block do.
      auto desc = [&](uint32_t base, bool mn, int plane_bytes, int p, int k16) {
        return mn ? make_smem_desc(base + p * (kBK * 128) + k16 * 2048, 3 * kBK * 128, 1024)
                  : make_smem_desc(base + p * plane_bytes + k16 * 32, 16, 1024);
      };
      auto product = [&](uint32_t tmem_d, uint32_t sa, uint32_t sb, int pa, int pb, bool first) {
#pragma unroll
        for (int k16 = 0; k16 < kBK / 16; ++k16)
          umma2_bf16(tmem_d, desc(sa, A_MN, Cfg::kAPlane, pa, k16), desc(sb, B_MN, Cfg::kBPlane, pb, k16), kIdesc,
                     first && k16 == 0 ? 0u : 1u);
      };
      auto commit_both = [&](uint64_t* bar) {
        const uint32_t a = smem_u32(bar);
        umma2_commit(a);
        umma2_commit(map_to_cta(a, 1));
      };
      int stage = 0, iter = 0, mi = 0;
      uint32_t phase = 0;
      bool alive = true;
      for (int unit = cluster_id; unit < total_units && alive; unit += n_clusters, ++iter) {
        const TileCtx t = decode_pair_tile(geom, unit, BN, 0);
        const int kb0 = t.split * geom.kb_per_split, kb1 = min(geom.k_blocks, kb0 + geom.kb_per_split);
        const int cb = iter % MB;
        for (int kb = kb0; kb < kb1; ++kb, ++mi) {
          const int mb = mi % MB;
          alive = mbar_wait(&full_bar[stage], phase, abort_flag, status, kStatusMmaTimeout) &&
                  mbar_wait(&mempty[mb], ((mi / MB) & 1u) ^ 1u, abort_flag, status, kStatusMmaTimeout);
          if (!alive) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + stage * Cfg::kStageBytes), sb = sa + 3 * Cfg::kAPlane;
          product(tmem_base + mb * BN, sa, sb, 0, 0, true);
          commit_both(&mfull[mb]);
          if (kb == kb0) {
            alive = mbar_wait(&cempty[cb], ((iter / MB) & 1u) ^ 1u, abort_flag, status, kStatusMmaTimeout);
            if (!alive) break;
            tc_fence_after();
          }
          const uint32_t small = tmem_small + cb * BN;
          product(small, sa, sb, 0, 2, kb == kb0);
          product(small, sa, sb, 2, 0, false);
          product(small, sa, sb, 1, 1, false);
          product(small, sa, sb, 0, 1, false);
          product(small, sa, sb, 1, 0, false);
          commit_both(&empty_bar[stage]);
          if (++stage == ST) stage = 0, phase ^= 1u;
        }
        if (alive) commit_both(&cfull[cb]);
      }
      if (!alive)
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs, own rows)
    constexpr int kChunks = BN / 64;  // 32-column chunks of this warp
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const bool planes_ok = !out.flags.any_in_warp(lane);
    int iter = 0, mi = 0;
    bool alive = true;
    for (int unit = cluster_id; unit < total_units && alive; unit += n_clusters, ++iter) {
      const TileCtx t = decode_pair_tile(geom, unit, BN, rank);
      const int kb0 = t.split * geom.kb_per_split, kb1 = min(geom.k_blocks, kb0 + geom.kb_per_split);
      float acc[kChunks][32];
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c][i] = 0.f;
      auto add = [&](uint32_t tmem) {
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
#pragma unroll
          for (int h = 0; h < 32; h += 16) {
            float v[16];
            tmem_ld16<0>(tmem + lanes + (2 * c + half) * 32 + h, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[c][h + i] += v[i];
          }
        }
        tc_fence_before();
        __syncwarp();
      };
      for (int kb = kb0; kb < kb1; ++kb, ++mi) {
        const int mb = mi % MB;
        alive = __all_sync(0xffffffffu,
                           mbar_wait(&mfull[mb], (mi / MB) & 1u, abort_flag, status, kStatusEpilogueTimeout));
        if (!alive) break;
        tc_fence_after();
        add(tmem_base + mb * BN);
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&mempty[mb]), 0));
      }
      if (!alive) break;
      const int cb = iter % MB;
      alive = __all_sync(0xffffffffu,
                         mbar_wait(&cfull[cb], (iter / MB) & 1u, abort_flag, status, kStatusEpilogueTimeout));
      if (!alive) break;
      tc_fence_after();
      add(tmem_small + cb * BN);
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&cempty[cb]), 0));
      const int row = quarter * 32 + lane;
      if (row >= t.rows_valid || !planes_ok) continue;
      float* dst = out.C + t.split * out.split_stride + static_cast<long long>(t.row0 + row) * out.ldc;
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const int col = t.col0 + (2 * c + half) * 32, left = geom.n_cols - col;
        float* d = dst + col;
        if (left >= 32 && (reinterpret_cast<uintptr_t>(d) & 15) == 0) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 v = make_float4(out.alpha * acc[c][4 * j], out.alpha * acc[c][4 * j + 1],
                                   out.alpha * acc[c][4 * j + 2], out.alpha * acc[c][4 * j + 3]);
            float4* q = reinterpret_cast<float4*>(d) + j;
            if (out.accumulate) {
              const float4 o = *q;
              v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
            }
            *q = v;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < left) {
              const float v = out.alpha * acc[c][i];
              d[i] = out.accumulate ? d[i] + v : v;
            }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512);
  }
}

// C (+)= alpha * sum over the K splits, in their order (the same bits on every run).
__global__ void __launch_bounds__(256) sum_splits_kernel(const float* __restrict__ part, float* __restrict__ C,
                                                         long long M, int N, int ldp, long long ldc, int splits,
                                                         float alpha, int accumulate, const SgemmFlags flags) {
  griddep_wait();
  griddep_launch();
  if (flags.any_in_block()) return;
  const int per_row = ldp / 4;
  const long long total = M * per_row, stride = M * ldp;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const long long r = i / per_row;
    const int c = static_cast<int>(i - r * per_row) * 4;
    float4 s = __ldg(reinterpret_cast<const float4*>(part + r * ldp + c));
    for (int k = 1; k < splits; ++k) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(part + k * stride + r * ldp + c));
      s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
    const float o[4] = {s.x, s.y, s.z, s.w};
    float* d = C + r * ldc + c;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c + e < N) d[e] = accumulate ? d[e] + alpha * o[e] : alpha * o[e];
  }
}

// ---------------------------------------------------------------------------- host side
struct F32Plan {
  int bn, split;
};

// Tile width and K split by estimated time in tensor cycles: waves of (tile, split) units over the 74 SM pairs, 3072
// cycles per k-block of a 256-wide tile (1536 at 128), about 2500 cycles per unit for filling the pipeline and storing,
// and, when K is split, a pass that adds the partial sums (4 bytes x (splits + 1) per output at about 2.5 KB a cycle,
// plus a launch).  Only accumulated products (weight gradients) are split: the additions of a plain product have one
// order whatever M is.
F32Plan pick_f32_plan(int64_t M, int64_t N, int64_t K, int out_mode) {
  const int64_t kb = ceil_div(K, kBK), slots = sm_count() / 2;
  F32Plan best{256, 1};
  double best_cost = -1.0;
  for (int bn = 256; bn >= 128; bn -= 128) {
    const int64_t units = ceil_div(M, 256) * ceil_div(N, bn);
    for (int64_t s = 1; s <= 16 && (s == 1 || (out_mode == POM_OUT_F32_ACCUM && kb / s >= kMinSplitBlocks)); ++s) {
      const int64_t per = ceil_div(kb, s), splits = ceil_div(kb, per);
      if (splits != s) continue;
      double cost = static_cast<double>(ceil_div(units * s, slots)) * (per * 12.0 * bn + 2500.0);
      if (s > 1) cost += 6000.0 + static_cast<double>(M) * N * 4.0 * (s + 1) / 2500.0;
      if (best_cost < 0 || cost < best_cost * 0.999) best_cost = cost, best = F32Plan{bn, static_cast<int>(s)};
    }
  }
  return best;
}

int plane_map(CUtensorMap* m, const void* planes, int64_t rows, int64_t cols, int box_cols, int box_rows) {
  const int64_t ld = plane_ld(cols);
  uint64_t dims[3] = {static_cast<uint64_t>(cols), static_cast<uint64_t>(rows), 3};
  uint64_t str[2] = {static_cast<uint64_t>(ld), static_cast<uint64_t>(ld * rows)};
  uint32_t box[3] = {static_cast<uint32_t>(box_cols), static_cast<uint32_t>(box_rows), 3};
  return make_map(m, planes, 3, dims, str, box);
}

template <int BN, bool A_MN, bool B_MN>
int launch_f32(const pom_gemm_args* a, const void* pa, const void* pb, int split, const F32Out& out, int* status,
               cudaStream_t st) {
  CUtensorMap tmA, tmB;
  int rc = A_MN ? plane_map(&tmA, pa, a->K, a->M, 64, kBK) : plane_map(&tmA, pa, a->M, a->K, kBK, kBM);
  if (rc) return rc;
  rc = B_MN ? plane_map(&tmB, pb, a->K, a->N, 64, kBK) : plane_map(&tmB, pb, a->N, a->K, kBK, BN / 2);
  if (rc) return rc;
  Operands o{a->A, a->Bm, a->M, a->N, a->K, 0, 0, 1, A_MN, B_MN};
  const GemmGeom g = make_geom(o, BN, split);
  auto kern = gemm_f32_planes_kernel<BN, A_MN, B_MN>;
  static std::atomic<uint64_t> attr_set{0};
  if ((rc = set_smem_once(kern, F32Cfg<BN>::kSmem, &attr_set))) return rc;
  const long long units = ceil_div(a->M, 256) * g.n_tiles * g.split_k;
  if (units > INT32_MAX) return POM_ERR_TOO_LARGE;
  const int clusters = static_cast<int>(units < sm_count() / 2 ? units : sm_count() / 2);
  if (launch_pdl(kern, dim3(2 * clusters), dim3(kF32Threads), F32Cfg<BN>::kSmem, st, tmA, tmB, g, out, status) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return POM_ERR_CUDA;
  }
  count_launch();
  return check_launch();
}

template <int BN>
int launch_f32_any(const pom_gemm_args* a, const void* pa, const void* pb, int split, const F32Out& out, int* status,
                   cudaStream_t st) {
  if (!a->a_mn_major && !a->b_mn_major) return launch_f32<BN, false, false>(a, pa, pb, split, out, status, st);
  if (!a->a_mn_major) return launch_f32<BN, false, true>(a, pa, pb, split, out, status, st);
  if (!a->b_mn_major) return launch_f32<BN, true, false>(a, pa, pb, split, out, status, st);
  return launch_f32<BN, true, true>(a, pa, pb, split, out, status, st);
}

SplitMat split_mat(const void* src, int64_t rows, int64_t cols, int64_t ld, void* planes) {
  SplitMat m;
  m.src = static_cast<const float*>(src);
  m.dst = reinterpret_cast<uint4*>(planes_of(planes));
  m.flags = static_cast<int*>(planes);
  m.rows = rows, m.cols = cols, m.ld = ld;
  m.groups = plane_ld(cols) / 8;
  m.blocks = split_blocks(rows, cols);
  return m;
}

// `norms` != NULL: the 2-norms of the rows of both operands (K-major, neither ready) are written there.
int planes_product(const pom_gemm_args* a, void* a_planes, int a_ready, void* b_planes, int b_ready, float* norms,
                   void* scratch, int* status, cudaStream_t st) {
  if (!a || !a->A || !a->Bm || !a->C || !a_planes || !b_planes) return POM_ERR_NULL;
  if (a->M <= 0 || a->N <= 0 || a->K <= 0) return POM_ERR_BAD_SHAPE;
  if (a->out_mode != POM_OUT_F32 && a->out_mode != POM_OUT_F32_ACCUM) return POM_ERR_UNSUPPORTED;
  if (a->batches != 1) return POM_ERR_UNSUPPORTED;
  if (ceil_div(a->M, 64) > 65535 || a->N > INT32_MAX || a->K > INT32_MAX) return POM_ERR_TOO_LARGE;  // as pom_gemm_f32
  if (!aligned16(a_planes) || !aligned16(b_planes) || !aligned16(scratch)) return POM_ERR_BAD_ALIGN;
  const int64_t ar = a->a_mn_major ? a->K : a->M, ac = a->a_mn_major ? a->M : a->K;
  const int64_t br = a->b_mn_major ? a->K : a->N, bc = a->b_mn_major ? a->N : a->K;
  SplitMat ma = split_mat(a->A, ar, ac, a->lda, a_planes), mb = split_mat(a->Bm, br, bc, a->ldb, b_planes);
  int log_k = 0;
  while ((1ll << log_k) < a->K) ++log_k;
  // exponent fields are 127 above the exponents of values times 2^24; a magnitude is below 2^(its exponent + 1)
  const SgemmFlags flags{ma.flags, ma.blocks, mb.flags, mb.blocks, 2 * 127 + 126 - 2 - log_k, 2 * 127 - 100};
  if (!a_ready || !b_ready) {
    const SplitMat& first = a_ready ? mb : ma;
    const int two = !a_ready && !b_ready;
    const int blocks = two && mb.blocks > ma.blocks ? mb.blocks : first.blocks;
    if ((norms ? launch_pdl(split_rows_kernel, dim3(blocks, 1 + two), dim3(kSplitThreads), 0, st, first, mb, norms)
               : launch_pdl(split_planes_kernel, dim3(blocks, 1 + two), dim3(kSplitThreads), 0, st, first, mb)) !=
        cudaSuccess) {
      (void)cudaGetLastError();
      return POM_ERR_CUDA;
    }
    count_launch();
  }
  const F32Plan plan = pick_f32_plan(a->M, a->N, a->K, a->out_mode);
  const int ldp = static_cast<int>((a->N + 3) / 4 * 4);
  const bool accumulate = a->out_mode == POM_OUT_F32_ACCUM;
  // an alpha that the planes' factor would make subnormal: the FMA kernel (with the planes in place for a later product)
  if (a->alpha != 0.f && fabsf(a->alpha) < 0x1p-78f) return launch_sgemm(a, SgemmFlags{nullptr, 0, nullptr, 0, 0, 0}, st);
  F32Out out{static_cast<float*>(a->C), a->ldc, 0, a->alpha * kUnscale, accumulate, flags};
  if (plan.split > 1) {
    if (!scratch) return POM_ERR_NULL;
    out = F32Out{static_cast<float*>(scratch), ldp, a->M * ldp, kUnscale, 0, flags};
  }
  const void *pa = planes_of(a_planes), *pb = planes_of(b_planes);
  const int rc = plan.bn == 256 ? launch_f32_any<256>(a, pa, pb, plan.split, out, status, st)
                                : launch_f32_any<128>(a, pa, pb, plan.split, out, status, st);
  if (rc) return rc;
  if (plan.split > 1) {
    const int64_t want = ceil_div(a->M * (ldp / 4), 256), cap = 8ll * sm_count();
    if (launch_pdl(sum_splits_kernel, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(256), 0, st,
                   static_cast<const float*>(scratch), static_cast<float*>(a->C), static_cast<long long>(a->M),
                   static_cast<int>(a->N), ldp, static_cast<long long>(a->ldc), plan.split, a->alpha,
                   static_cast<int>(accumulate), flags) != cudaSuccess) {
      (void)cudaGetLastError();
      return POM_ERR_CUDA;
    }
    count_launch();
  }
  // operands that the planes cannot carry: the FMA kernel, whose blocks return at once when no flag is up
  return launch_sgemm(a, flags, st);
}

}  // namespace

extern "C" {

uint64_t pom_f32_planes_bytes(int64_t rows, int64_t cols) {
  if (rows <= 0 || cols <= 0) return 0;
  return kFlagBytes + 3ull * static_cast<uint64_t>(rows) * static_cast<uint64_t>(plane_ld(cols)) * 2ull;
}

uint64_t pom_gemm_f32_planes_scratch(int64_t M, int64_t N, int64_t K, int32_t out_mode) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const F32Plan p = pick_f32_plan(M, N, K, out_mode);
  return p.split > 1 ? static_cast<uint64_t>(p.split) * M * ((N + 3) / 4 * 4) * 4 : 0;
}

int pom_gemm_f32_planes(const pom_gemm_args* a, void* a_planes, int a_ready, void* b_planes, int b_ready, void* scratch,
                        int* status, void* stream) {
  return planes_product(a, a_planes, a_ready, b_planes, b_ready, nullptr, scratch, status,
                        static_cast<cudaStream_t>(stream));
}

int pom_project_f32(const pom_gemm_args* a, void* a_planes, void* b_planes, float* norms, int64_t gate_col0,
                    const float* gate_bias, int* status, void* stream) {
  if (!a || !norms) return POM_ERR_NULL;
  if (a->a_mn_major || a->b_mn_major || a->out_mode != POM_OUT_F32 || a->alpha != 1.f) return POM_ERR_UNSUPPORTED;
  if (gate_col0 < 0 || gate_col0 > a->N) return POM_ERR_BAD_SHAPE;
  if (gate_col0 < a->N && !gate_bias) return POM_ERR_NULL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = planes_product(a, a_planes, 0, b_planes, 0, norms, nullptr, status, st);
  if (rc) return rc;
  NearArgs n;
  n.A = static_cast<const float*>(a->A), n.B = static_cast<const float*>(a->Bm), n.C = static_cast<float*>(a->C);
  n.norms = norms, n.bias = gate_bias;
  n.lda = a->lda, n.ldb = a->ldb, n.ldc = a->ldc;
  n.M = static_cast<int>(a->M), n.N = static_cast<int>(a->N), n.K = static_cast<int>(a->K);
  n.gate0 = static_cast<int>(gate_col0);
  n.factor = 8.f * sqrtf(static_cast<float>(a->K)) * 0x1p-24f;
  const int64_t want = ceil_div(a->M * ((a->N + 3) / 4), 256), cap = 8ll * sm_count();
  if (launch_pdl(near_kinks_kernel, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(256), 0, st, n) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return POM_ERR_CUDA;
  }
  count_launch();
  return check_launch();
}
}  // extern "C"
