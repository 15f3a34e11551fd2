#include "nvl/nvl_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickKernelT<double>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
