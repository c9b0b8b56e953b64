// FP32 factorisation + FP64 refinement instantiations of the latency kernel (eight warps per mode).
#include "sbz_pt_lat.cuh"

namespace sbz {

int pt_launch_lat_f32(const PtArgs& A, int num_sms, cudaStream_t stream) {
  switch ((A.model_n + ptk::kSolvers - 1) / ptk::kSolvers) {
    case 1: return ptk::launch_lat<1, float>(A, num_sms, stream);
    case 2: return ptk::launch_lat<2, float>(A, num_sms, stream);
    default: return SBZ_ERR_ARG;
  }
}

}  // namespace sbz
