#include "mega_launch.cuh"

namespace cd {
template cudaError_t launch_mega<__nv_bfloat16, Fp8Row, __half>(cd_model*, int, int);
template cudaError_t launch_mega<__nv_bfloat16, Fp8Row, __nv_bfloat16>(cd_model*, int, int);
}  // namespace cd
