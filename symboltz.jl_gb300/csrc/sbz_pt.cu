// Precision and group-size dispatch of the perturbation kernel (sbz_pt_impl.cuh).
#include "sbz_pt.cuh"

namespace sbz {

int pt_launch_f32_w1(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_f32_w2_w4(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_f64_w1(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_f64_w2_w4(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_lat_f32(const PtArgs& A, int num_sms, cudaStream_t stream);
int pt_launch_lat_f64(const PtArgs& A, int num_sms, cudaStream_t stream);
int pt_launch_thr_f32(const PtArgs& A, int modes_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_thr_f64(const PtArgs& A, int modes_per_sm, int num_sms, cudaStream_t stream);

// Warps per mode when the caller leaves it open.  The results of a mode depend on it (order of the norms'
// sums, refinement default), not on the kernel that runs it.
static int auto_warps_per_mode(int nitems, int num_sms) { return nitems <= 32 * num_sms ? 4 : 1; }

// Modes that share an SM when the caller leaves it open, 1: the latency kernel.  A launch lasts as long as
// the slower of its longest mode and its total work over the SMs: with few modes per SM to go round, each
// gets an SM's FP64 pipes to itself, with many they share them (times in sbz_pt_thr.cuh).  The lines are
// where the curves of neighbouring shapes cross for k up to 0.05 .. 1 h/Mpc: 1,040 modes of n = 47 take 62.6
// ms one per SM and 56.8 two per SM, of n = 133 75.9 and 76.2; 1,328 against 1,600 two or three per SM; 2,400
// against 3,200 three or four; 4,800 four or eight.
static int thr_modes_per_sm(int nitems, int n, int num_sms) {
  const int q = (nitems + num_sms - 1) / num_sms;
  return q <= (n > 96 ? 7 : 6) ? 1 : q <= 9 ? 2 : q <= 15 ? 3 : q <= 28 ? 4 : 8;
}

int pt_launch(const PtArgs& A, int precision, int warps_per_block, int warps_per_mode, int blocks_per_sm, int num_sms,
              cudaStream_t stream) {
  if (warps_per_block <= 0) warps_per_block = 4;
  const bool open_blocks = blocks_per_sm <= 0;
  const int nw = warps_per_mode > 0 ? warps_per_mode : auto_warps_per_mode(A.nitems, num_sms);
  if (nw != 1 && nw != 2 && nw != 4 && nw != 8) return SBZ_ERR_ARG;
  const int modes = thr_modes_per_sm(A.nitems, A.model_n, num_sms);
  // throughput kernel: blocks left open, chains that fit a warp; one-warp modes only where the width was
  // left open too (asked for, they keep their own kernel)
  const bool thr = open_blocks && modes > 1 && A.chain_rows <= 32 && (warps_per_mode <= 0 || nw == 2 || nw == 4);
  if (blocks_per_sm <= 0 && nw == 4) blocks_per_sm = A.nitems <= 8 * num_sms ? 1 : 2;
  if (nw == 8) blocks_per_sm = 1;  // eight-warp groups: one mode per SM
  // latency kernel: one mode per SM, while its four solver warps hold every chain (nx <= 5)
  const bool lat = !thr && nw == 4 && blocks_per_sm == 1 && A.nchain <= 8 && A.chain_rows <= 32;
  if (precision == SBZ_MIXED) {
    // lazy refinement left open: the later stages skip their FP64 refinement when stage 1's first
    // correction is below 1e-5 error weights (Rodas5P's stage right-hand sides carry coefficients up
    // to 165, so an unrefined FP32 stage solve stays below the refinement's own 1e-3 stopping level
    // only when stage 1's was well below 1e-5); on for four-warp groups (latency-bound), off for
    // narrower ones (throughput-bound batches).  Skipping the later stages' refinement outright was
    // measured to leave pointwise sources 0.48 (rtol 1e-5) and 1.1e-2 (rtol 1e-7) of their maximum
    // away from the oracle on the reference's ΛCDM(lmax = 5) model.
    PtArgs B = A;
    if (B.refine_skip < 0) B.refine_skip = nw >= 4 ? 1e-5f : 0.0f;
    B.norm_warps = nw;
    if (thr) return pt_launch_thr_f32(B, modes, num_sms, stream);
    if (lat) return pt_launch_lat_f32(B, num_sms, stream);
    return nw == 1 ? pt_launch_f32_w1(B, nw, warps_per_block, blocks_per_sm, num_sms, stream)
                   : pt_launch_f32_w2_w4(B, nw, warps_per_block, blocks_per_sm, num_sms, stream);
  }
  PtArgs B = A;
  B.norm_warps = nw;
  if (thr) return pt_launch_thr_f64(B, modes, num_sms, stream);
  if (lat) return pt_launch_lat_f64(A, num_sms, stream);
  return nw == 1 ? pt_launch_f64_w1(A, nw, warps_per_block, blocks_per_sm, num_sms, stream) : pt_launch_f64_w2_w4(A, nw, warps_per_block, blocks_per_sm, num_sms, stream);
}

}  // namespace sbz
