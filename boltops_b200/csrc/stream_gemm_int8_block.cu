// Weight-streaming grouped GEMM, block-scaled int8 operands (stream_gemm.cuh).
#include "stream_gemm.cuh"

namespace bolt {
namespace stream {
BOLT_STREAM_DEFINE(OP_I8, true)
}  // namespace stream
}  // namespace bolt
