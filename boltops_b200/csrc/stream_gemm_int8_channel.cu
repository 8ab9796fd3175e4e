// Weight-streaming grouped GEMM, per-channel int8 operands (stream_gemm.cuh).
#include "stream_gemm.cuh"

namespace bolt {
namespace stream {
BOLT_STREAM_DEFINE(OP_I8, false)
}  // namespace stream
}  // namespace bolt
