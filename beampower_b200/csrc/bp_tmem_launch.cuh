// Launch dispatch of the tensor-memory kernel (template bodies).  Included only
// by the bp_tmem_*.cu files, each of which instantiates one (storage, reduce).
#pragma once

#include <algorithm>

#define BP_TEMPLATE_KERNELS_ONLY
#include "bp_host.h"
#include "bp_tmem.cuh"

namespace bp_host {

template <int P, bool MAXRED, int STORAGE>
int launch_tmem_p(bp::LaunchArgs a, bool batch, long long plain_blocks, int dev,
                  cudaStream_t st) {
  const bp::TmLayout lay = bp::tm_layout<P, MAXRED>(a.rowcap, a.max_active, a.n_stage);
  a.tm = lay;
  if (lay.total > (size_t)device_smem_optin(dev))
    return fail(BP_ERR_UNSUPPORTED, "tensor-memory kernel needs %u B of shared memory", lay.total);
  if (batch) {
    if constexpr (MAXRED) {
      auto kern = bp::beam_tmem_batch_kernel<P, STORAGE>;
      BP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)lay.total));
      kern<<<std::max(1, device_sm_count(dev)), bp::kTmThreads, lay.total, st>>>(a);
      BP_LAUNCHED("beam_tmem_batch_kernel");
    }
    return BP_OK;
  }
  const bool share = a.tiles_per_chunk == 0;  // a block per SM, equal shares
  auto kern = share ? bp::beam_tmem_share_kernel<P, MAXRED, STORAGE>
                    : bp::beam_tmem_kernel<P, MAXRED, STORAGE>;
  BP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)lay.total));
  if (plain_blocks > kMaxInt) return fail(BP_ERR_UNSUPPORTED, "grid too large");
  if (plain_blocks <= 0) return BP_OK;
  kern<<<(unsigned)plain_blocks, bp::kTmThreads, lay.total, st>>>(a);
  BP_LAUNCHED("tensor-memory kernel");
  return BP_OK;
}

template <bool MAXRED, int STORAGE>
int launch_tmem(int P, const bp::LaunchArgs& a, bool batch, long long blocks, int dev,
                cudaStream_t st) {
  switch (P) {
    case 1: return launch_tmem_p<1, MAXRED, STORAGE>(a, batch, blocks, dev, st);
    case 2: return launch_tmem_p<2, MAXRED, STORAGE>(a, batch, blocks, dev, st);
    case 3: return launch_tmem_p<3, MAXRED, STORAGE>(a, batch, blocks, dev, st);
    case 4: return launch_tmem_p<4, MAXRED, STORAGE>(a, batch, blocks, dev, st);
    default: return fail(BP_ERR_UNSUPPORTED, "tensor-memory kernel supports 1..4 phases");
  }
}

}  // namespace bp_host
