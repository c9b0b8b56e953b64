// all-FP64 instantiations of the throughput kernel, four warps per mode.
#include "sbz_pt_thr.cuh"

namespace sbz {

int pt_launch_thr2_f64(const PtArgs& A, int num_sms, cudaStream_t stream);

int pt_thr2_resident_f64(int n) { return ptk::thr2_resident<double>(n); }

int pt_launch_thr_f64(const PtArgs& A, int warps, int modes_per_sm, int num_sms, cudaStream_t stream) {
  using namespace ptk;
  if (warps == 2) return pt_launch_thr2_f64(A, num_sms, stream);
  const int slots = (A.model_n + 127) / 128;
  if (slots < 1 || slots > 2) return SBZ_ERR_ARG;
  if (modes_per_sm > 3) return slots == 1 ? launch_thr<4, 256, 2, 1, double>(A, 2, num_sms, stream) : SBZ_ERR_ARG;  // above 107 equations four have two warps
  return slots == 1 ? launch_thr<4, 128, 3, 1, double>(A, modes_per_sm, num_sms, stream)
                    : launch_thr<4, 128, 3, 2, double>(A, modes_per_sm, num_sms, stream);
}

}  // namespace sbz
