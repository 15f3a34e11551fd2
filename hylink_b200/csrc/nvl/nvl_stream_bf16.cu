#include "nvl/nvl_stream_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickStreamT<__nv_bfloat16>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
