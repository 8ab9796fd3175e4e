// Host side of the weight-streaming grouped GEMM (kernel and description: stream_gemm.cuh).
#include "stream_gemm.cuh"

namespace bolt {
namespace stream {
BOLT_STREAM_KINDS(BOLT_STREAM_EXTERN)
}  // namespace stream

int stream_gemm(const bolt_gemm_args* a, const CUtensorMap& mb, cudaStream_t st) {
  using namespace stream;
  using tc::OP_F16;
  using tc::OP_F8;
  using tc::OP_I8;
  const bool gated = a->epilogue != BOLT_EPI_STORE;
  const bool is16 = a->kind == BOLT_GEMM_BF16 || a->kind == BOLT_GEMM_F16;
  const bool block = a->kind == BOLT_GEMM_FP8_BLOCK || a->kind == BOLT_GEMM_INT8_BLOCK;
  const int elem = is16 ? 2 : 1;
  StreamParams p{};
  p.a = a->a;
  p.a_row_bytes = a->a_gather && a->a_row_bytes > 0 ? a->a_row_bytes : (int64_t)a->k * elem;
  p.a_scale = a->a_scale;
  p.a_scale_ld = a->a_scale_ld;
  p.b_scale = a->b_scale;
  p.bias = a->bias;
  p.bias_dtype = a->bias_dtype;
  p.c = a->c;
  p.c_dtype = a->c_dtype;
  p.mid_dtype = a->mid_dtype;
  p.c_ld = a->c_ld;
  p.c_scale = a->c_scale;
  p.c_scale_ld = a->c_scale_ld;
  p.gather = a->a_gather != 0;
  p.a_scale_tok = a->a_scale_token_order;
  p.scatter = a->scatter;
  p.num_tokens = a->num_tokens;
  p.topk = a->topk;
  p.mul_routed_weight = a->mul_routed_weight;
  p.c_vec_ok = reinterpret_cast<uintptr_t>(a->c) % 16 == 0 &&
               (a->c_ld * (int64_t)dtype_bytes(a->c_dtype)) % 16 == 0;
  p.sorted_ids = a->sorted_ids;
  p.sorted_weights = a->sorted_weights;
  p.expert_ids = a->sorted_expert_ids;
  p.num_valid = a->num_valid_ids;
  p.status = a->status;
  p.n = a->n;
  p.n_half = a->n / 2;
  p.num_experts = a->num_experts;
  p.capacity = a->capacity;
  p.num_kb = a->k * elem / 128;
  p.kb_scale_cols = a->k / 128;

  const bool is_int = a->kind == BOLT_GEMM_INT8_CHANNEL || a->kind == BOLT_GEMM_INT8_BLOCK;
  const uint32_t fmt = a->kind == BOLT_GEMM_BF16 || is_int ? 1u : 0u;
  p.idesc = ((is_int ? 2u : 1u) << 4) | (fmt << 7) | (fmt << 10) | ((128u >> 4) << 24);

  const int sms = a->sm_count > 0 ? a->sm_count : sm_count_of_current_device();
  // Items: plain ones of the kinds that sum over K in TMEM are halved while whole ones leave CTAs
  // with fewer than four each (a row tile per touched expert at most) and no tile needs a second pass
  // over the weights (half an item holds 64 rows; only tokens that name an expert twice make more).  A gated item needs its gate half and its up
  // half, and the block-scaled kinds would hand TMEM stages over twice as often per byte.
  // Measured, down projection: Mixtral bf16 with one token 110 -> 65 us, with 23 tokens 149 us either
  // way, DeepSeek-V3 fp8 with 96 tokens 545 -> 717 us.
  const int64_t routes = (int64_t)a->num_tokens * a->topk;
  const int64_t row_tiles = routes < a->num_experts ? routes : a->num_experts;
  const int cols = gated ? a->n / 2 : a->n;
  int width = gated ? 128 : 256;
  const int kbs = !gated && !block && a->num_tokens <= kMaxRows / 2 &&
                          row_tiles * ((cols + width - 1) / width) < 4ll * sms
                      ? 2
                      : 1;
  width /= kbs;
  p.tiles_n = (cols + width - 1) / width;
  const int64_t max_items = (int64_t)(a->capacity / 128) * p.tiles_n;
  const int grid = (int)(max_items < sms ? max_items : sms);
  switch (a->kind) {
    case BOLT_GEMM_BF16:
    case BOLT_GEMM_F16: return launch_kind<OP_F16, false>(a->epilogue, kbs, mb, p, grid, st);
    case BOLT_GEMM_FP8_BLOCK: return launch_kind<OP_F8, true>(a->epilogue, kbs, mb, p, grid, st);
    case BOLT_GEMM_FP8_CHANNEL: return launch_kind<OP_F8, false>(a->epilogue, kbs, mb, p, grid, st);
    case BOLT_GEMM_INT8_CHANNEL: return launch_kind<OP_I8, false>(a->epilogue, kbs, mb, p, grid, st);
    case BOLT_GEMM_INT8_BLOCK: return launch_kind<OP_I8, true>(a->epilogue, kbs, mb, p, grid, st);
    default: break;
  }
  set_error("grouped_gemm: unsupported kind %d", a->kind);
  return BOLT_ERR_UNSUPPORTED;
}

}  // namespace bolt
