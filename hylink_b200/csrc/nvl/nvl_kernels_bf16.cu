#include "nvl/nvl_kernels.cuh"

namespace hl {
namespace nvl {
template const void* pickKernelT<__nv_bfloat16>(int kind, int nranks);
}  // namespace nvl
}  // namespace hl
