// Tensor-memory kernel variants of bf16 storage, whole response.
#include "bp_tmem_launch.cuh"

namespace bp_host {
template int launch_tmem<false, BP_STORAGE_BF16>(int, const bp::LaunchArgs&, bool, long long, int,
                                               cudaStream_t);
}  // namespace bp_host
