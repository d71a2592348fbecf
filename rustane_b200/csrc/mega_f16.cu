#include "mega_launch.cuh"

namespace cd {
template cudaError_t launch_mega<__half, __half, __half>(cd_model*, int, int);
}  // namespace cd
