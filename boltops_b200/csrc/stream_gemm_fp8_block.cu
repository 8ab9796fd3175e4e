// Weight-streaming grouped GEMM, block-scaled e4m3 operands (stream_gemm.cuh).
#include "stream_gemm.cuh"

namespace bolt {
namespace stream {
BOLT_STREAM_DEFINE(OP_F8, true)
}  // namespace stream
}  // namespace bolt
