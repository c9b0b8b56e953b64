// all-FP64 instantiations of the latency kernel (eight warps per mode).
#include "sbz_pt_lat.cuh"

namespace sbz {

int pt_launch_lat_f64(const PtArgs& A, int num_sms, cudaStream_t stream) {
  switch ((A.model_n + ptk::kSolvers - 1) / ptk::kSolvers) {
    case 1: return ptk::launch_lat<1, double>(A, num_sms, stream);
    case 2: return ptk::launch_lat<2, double>(A, num_sms, stream);
    default: return SBZ_ERR_ARG;
  }
}

}  // namespace sbz
