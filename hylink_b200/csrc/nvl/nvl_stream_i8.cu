#include "nvl/nvl_stream_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickStreamT<int8_t>(int kind, int nranks);
template const void* pickStreamT<uint8_t>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
