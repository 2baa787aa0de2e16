// Host launchers for the tcgen05 GEMM engine and its fused PoM epilogues.
#include <cudaTypedefs.h>
#include <mutex>
#include "common.cuh"
#include "epilogues.cuh"
#include "gemm_launch.cuh"

using namespace pomk;
using namespace pomh;

namespace pomh {
std::atomic<long long> g_launches{0};
// 0: automatic choice, 1: always the one-CTA kernel, 2: always the two-CTA (pair) kernel.
std::atomic<int> g_gemm_mode{0};
}

namespace pomh {

int gemm_bf16_dead_k(const pom_gemm_args* a, const float* tile_weight, int dead_k, int* status, cudaStream_t st) {
  if (!a || !a->C) return POM_ERR_NULL;
  Operands o{a->A, a->Bm, a->M, a->N, a->K, a->lda, a->ldb, a->batches, a->a_mn_major != 0, a->b_mn_major != 0};
  o.a_batch_stride = a->a_batch_stride;
  o.b_batch_stride = a->b_batch_stride;
  o.b_batched = a->b_batched != 0;
  o.tile_weight = dead_k > 0 ? tile_weight : nullptr;
  o.dead_k = dead_k;
  if (a->a_batch_stride % 8 || a->b_batch_stride % 8 || a->a_batch_stride < 0 || a->b_batch_stride < 0 ||
      a->c_batch_stride < 0)
    return POM_ERR_BAD_STRIDE;
  int rc = check_operands(o);
  if (rc) return rc;
  if (a->out_mode < 0 || a->out_mode > 2) return POM_ERR_UNSUPPORTED;
  if (a->ldc < a->N) return POM_ERR_BAD_STRIDE;
  if (a->out_mode == POM_OUT_BF16 && (a->ldc % 8 || !aligned16(a->C))) return POM_ERR_BAD_ALIGN;
  int split = a->split_k;
  if (a->out_mode != POM_OUT_F32_ACCUM) {
    if (split > 1) return POM_ERR_UNSUPPORTED;
    split = 1;
  }
  const TilePlan plan = pick_plan(o, true, a->out_mode == POM_OUT_F32_ACCUM && a->split_k == 0);
  if (split == 0) split = pick_split(plan_units(o, plan), ceil_div(a->K, kBK), plan.pair ? sm_count() / 2 : sm_count());
  EpiStore::Params ep;
  ep.C = a->C;
  ep.ldc = a->ldc;
  ep.batch_stride = a->c_batch_stride ? a->c_batch_stride : a->M * a->ldc;
  if (a->out_mode == POM_OUT_BF16 && a->c_batch_stride % 8) return POM_ERR_BAD_STRIDE;
  if (a->residual && a->c_batch_stride) return POM_ERR_UNSUPPORTED;
  ep.mode = a->out_mode;
  ep.alpha = a->alpha;
  ep.act = a->act;
  ep.residual = static_cast<const __nv_bfloat16*>(a->residual);
  ep.ldr = a->ldr;
  if ((a->act || a->residual) && a->out_mode != POM_OUT_BF16) return POM_ERR_UNSUPPORTED;
  if (a->act < 0 || a->act > 1 || (a->residual && a->ldr < a->N)) return POM_ERR_UNSUPPORTED;
  EpiMaps maps{};
  if (a->out_mode == POM_OUT_BF16 &&
      (rc = make_io_map(&maps.out0, a->C, a->N, a->M, a->batches, a->ldc, a->c_batch_stride)))
    return rc;
  return run_plan_any_major<EpiStore>(plan, o, split, maps, ep, status, st);
}

}  // namespace pomh

// =========================================================================== C ABI
extern "C" {

int pom_gemm_bf16(const pom_gemm_args* a, int* status, void* stream) {
  return gemm_bf16_dead_k(a, nullptr, 0, status, static_cast<cudaStream_t>(stream));
}

int pom_set_gemm_mode(int mode) {
  if (mode < 0 || mode % 10 > 2 || (mode / 10) % 10 > 3 || mode / 100 > 1) return POM_ERR_UNSUPPORTED;
  g_gemm_mode.store(mode);
  return POM_OK;
}

int pom_ctx_gemm(const pom_ctx_args* a, int* status, void* stream) {
  if (!a || !a->coeff || (!a->partial && !a->causal)) return POM_ERR_NULL;
  if (a->K < 1) return POM_ERR_BAD_SHAPE;
  if (a->causal) return ctx_gemm_causal(a, status, static_cast<cudaStream_t>(stream));
  if (a->rope.kind != POM_ROPE_NONE) return ctx_gemm_rope(a, status, static_cast<cudaStream_t>(stream));
  Operands o{a->X, a->Wpo, a->N, a->P, a->D, a->ldx, a->ldw, a->B, false, false};
  o.tile_weight = a->row_weight ? a->tile_weight : nullptr;
  int rc = check_operands(o);
  if (rc) return rc;
  if (a->hp_out && (a->ld_hp % 8 || a->ld_hp < a->P || !aligned16(a->hp_out))) return POM_ERR_BAD_ALIGN;
  EpiCtx::Params ep;
  ep.coeff = a->coeff;
  ep.K = a->K;
  ep.row_weight = a->row_weight;
  ep.save_hp = a->hp_out != nullptr;
  ep.partial = a->partial;
  ep.P = a->P;
  EpiMaps maps{};
  if (a->hp_out && (rc = make_io_map(&maps.out0, a->hp_out, a->P, a->N, a->B, a->ld_hp))) return rc;
  return run_plan<false, false, EpiCtx>(pick_plan(o, false), o, 1, maps, ep, status,
                                        static_cast<cudaStream_t>(stream));
}

int pom_gate_gemm(const pom_gate_args* a, int* status, void* stream) {
  if (!a || !a->bias || (!a->H && !a->causal) || !a->sh_out) return POM_ERR_NULL;
  if (a->causal) return gate_gemm_causal(a, status, static_cast<cudaStream_t>(stream));
  if (a->rope.kind != POM_ROPE_NONE) return gate_gemm_rope(a, status, static_cast<cudaStream_t>(stream));
  Operands o{a->X, a->Wse, a->T, a->P, a->D, a->ldx, a->ldw, a->B, false, false};
  int rc = check_operands(o);
  if (rc) return rc;
  if (a->h_row_stride != 0) return POM_ERR_UNSUPPORTED;
  if (a->ld_sh % 8 || a->ld_sh < a->P || !aligned16(a->sh_out)) return POM_ERR_BAD_ALIGN;
  if (a->z_out && (a->ld_z % 8 || a->ld_z < a->P || !aligned16(a->z_out))) return POM_ERR_BAD_ALIGN;
  EpiGate::Params ep;
  ep.bias = a->bias;
  ep.H = a->H;
  ep.h_batch_stride = a->h_batch_stride;
  ep.save_z = a->z_out != nullptr;
  EpiMaps maps{};
  if (a->z_out && (rc = make_io_map(&maps.out0, a->z_out, a->P, a->T, a->B, a->ld_z))) return rc;
  if ((rc = make_io_map(&maps.out1, a->sh_out, a->P, a->T, a->B, a->ld_sh))) return rc;
  return run_plan<false, false, EpiGate>(pick_plan(o, false), o, 1, maps, ep, status,
                                         static_cast<cudaStream_t>(stream));
}

int pom_gate_bwd_gemm(const pom_gate_bwd_args* a, int* status, void* stream) {
  if (!a || !a->bias || !a->z || !a->g_out || !a->db_partial) return POM_ERR_NULL;
  if (a->causal) return gate_bwd_gemm_causal(a, status, static_cast<cudaStream_t>(stream));
  if (!a->H || !a->dh_partial) return POM_ERR_NULL;
  if (a->rope.kind != POM_ROPE_NONE) return gate_bwd_gemm_rope(a, status, static_cast<cudaStream_t>(stream));
  // dSH[t, p] = sum_d dY[t, d] * Wo[d, p]: the B operand is Wo stored (K = D rows, N = P columns).
  Operands o{a->dY, a->Wo, a->T, a->P, a->D, a->ld_dy, a->ldw, a->B, false, true};
  int rc = check_operands(o);
  if (rc) return rc;
  if (a->ld_g % 8 || !aligned16(a->g_out) || a->ld_z % 8 || !aligned16(a->z)) return POM_ERR_BAD_ALIGN;
  EpiGateBwd::Params ep;
  ep.bias = a->bias;
  ep.H = a->H;
  ep.h_batch_stride = a->h_batch_stride;
  ep.dh_partial = a->dh_partial;
  ep.db_partial = a->db_partial;
  ep.P = a->P;
  EpiMaps maps{};
  if ((rc = make_io_map(&maps.in0, a->z, a->P, a->T, a->B, a->ld_z))) return rc;
  if ((rc = make_io_map(&maps.out0, a->g_out, a->P, a->T, a->B, a->ld_g))) return rc;
  return run_plan<false, true, EpiGateBwd>(pick_plan(o, false), o, 1, maps, ep, status,
                                           static_cast<cudaStream_t>(stream));
}

}  // extern "C"
