// FP32 factorisation + FP64 refinement instantiations of the throughput kernel, two warps per mode.
#include "sbz_pt_thr.cuh"

namespace sbz {

int pt_launch_thr2_f32(const PtArgs& A, int num_sms, cudaStream_t stream) {
  using namespace ptk;
  switch ((A.model_n + 63) / 64) {
    case 1: return launch_thr<2, 256, 2, 1, float>(A, 2, num_sms, stream);
    case 2: return launch_thr<2, 256, 2, 2, float>(A, 2, num_sms, stream);
    case 3: return launch_thr<2, 256, 2, 3, float>(A, 2, num_sms, stream);
    default: return SBZ_ERR_ARG;
  }
}

}  // namespace sbz
