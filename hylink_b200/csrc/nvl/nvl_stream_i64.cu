#include "nvl/nvl_stream_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickStreamT<long long>(int kind, int nranks);
template const void* pickStreamT<unsigned long long>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
