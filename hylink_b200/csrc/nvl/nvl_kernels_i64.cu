#include "nvl/nvl_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickKernelT<long long>(int kind, int nranks);
template const void* pickKernelT<unsigned long long>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
