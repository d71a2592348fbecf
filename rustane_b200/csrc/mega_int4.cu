#include "mega_launch.cuh"

namespace cd {
template cudaError_t launch_mega<__nv_bfloat16, Int4G32, __half>(cd_model*, int, int);
template cudaError_t launch_mega<__nv_bfloat16, Int4G32, __nv_bfloat16>(cd_model*, int, int);
}  // namespace cd
