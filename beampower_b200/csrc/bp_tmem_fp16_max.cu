// Tensor-memory kernel variants of fp16 storage, max/argmax reduction.
#include "bp_tmem_launch.cuh"

namespace bp_host {
template int launch_tmem<true, BP_STORAGE_F16>(int, const bp::LaunchArgs&, bool, long long, int,
                                               cudaStream_t);
}  // namespace bp_host
