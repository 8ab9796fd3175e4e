// Weight-streaming grouped GEMM, bf16 / fp16 operands (stream_gemm.cuh).
#include "stream_gemm.cuh"

namespace bolt {
namespace stream {
BOLT_STREAM_DEFINE(OP_F16, false)
}  // namespace stream
}  // namespace bolt
