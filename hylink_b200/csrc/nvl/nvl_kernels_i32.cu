#include "nvl/nvl_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickKernelT<int32_t>(int kind, int nranks);
template const void* pickKernelT<uint32_t>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
