// Tensor-memory kernel variants of fp32 storage, whole response.
#include "bp_tmem_launch.cuh"

namespace bp_host {
template int launch_tmem<false, BP_STORAGE_F32>(int, const bp::LaunchArgs&, bool, long long, int,
                                               cudaStream_t);
}  // namespace bp_host
