// Weight-streaming grouped GEMM, per-channel e4m3 operands (stream_gemm.cuh).
#include "stream_gemm.cuh"

namespace bolt {
namespace stream {
BOLT_STREAM_DEFINE(OP_F8, false)
}  // namespace stream
}  // namespace bolt
