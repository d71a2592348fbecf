#include "mega_launch.cuh"

namespace cd {
template cudaError_t launch_mega<float, float, float>(cd_model*, int, int);
}  // namespace cd
