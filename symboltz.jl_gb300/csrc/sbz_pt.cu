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

// Modes that share an SM when the caller leaves it open, 1: the latency kernel.  With few modes per SM to go
// round, each gets an SM's FP64 pipes to itself, with many they share them: a mode then takes `slow` times as
// long, but `modes` of them run at once.  A launch lasts about as long as the slower of its longest mode and its
// work over the SMs, slow · max(1, r / modes) in units of the longest mode alone on an SM, with
// r = Σ steps / (longest's steps · SMs).  The table holds the longest mode's measured times (ms, k up to
// 0.2 h/Mpc) over its time alone: mixed n = 47 38, 56, 61, 72, 107; n = 82
// 38.5, 56, 62, 77, 142; n = 133 45, 79, 89, 107, 170; FP64 n = 38 54, 71, 81, 100, 155; n = 133 (k up to 0.05)
// 20, 38, 51, 60, 73.  Lines on the mode count alone gave up to 40 %
// away where the modes' lengths are close (n = 133, k up to 0.02, 1,200 modes: two per SM 34.0 ms, four 24.7; n = 47, k
// up to 0.1 with 100 saved times, 912 modes: one 53.5, two 38.0); over 600 to 4,900 modes, k up to 0.02 .. 1 h/Mpc, with
// and without saved times and in FP64, this choice is within 10 % of the best shape (FP64 n = 133 at 800
// to 1,400 modes: 30 %).
static int thr_modes_per_sm(const PtArgs& A, int precision, int num_sms) {
  static const int modes[5] = {1, 2, 3, 4, 8};
  static const float mixed[3][5] = {{1, 1.45f, 1.56f, 1.87f, 2.8f}, {1, 1.45f, 1.61f, 2.0f, 3.7f}, {1, 1.75f, 1.96f, 2.35f, 3.75f}};
  static const float fp64[2][5] = {{1, 1.32f, 1.51f, 1.85f, 2.9f}, {1, 1.9f, 2.6f, 3.0f, 3.7f}};
  const float* slow = precision == SBZ_MIXED ? mixed[A.model_n <= 64 ? 0 : A.model_n <= 96 ? 1 : 2] : fp64[A.model_n <= 96 ? 0 : 1];
  const double r = (A.load > 0 ? A.load : 0.25 * A.nitems) / num_sms;  // modes on the device only: as of a geometric grid up to 0.2 h/Mpc
  int best = 0;
  double tb = r > 1 ? r : 1;
  for (int i = 1; i < 5; ++i) {
    const double t = slow[i] * (r > modes[i] ? r / modes[i] : 1);
    if (t < 0.99 * tb) { best = i; tb = t; }
  }
  return modes[best];
}

int pt_launch(const PtArgs& A, int precision, int warps_per_block, int warps_per_mode, int blocks_per_sm, int num_sms,
              cudaStream_t stream) {
  if (warps_per_block <= 0) warps_per_block = 4;
  const bool open_blocks = blocks_per_sm <= 0;
  const int nw = warps_per_mode > 0 ? warps_per_mode : auto_warps_per_mode(A.nitems, num_sms);
  if (nw != 1 && nw != 2 && nw != 4 && nw != 8) return SBZ_ERR_ARG;
  const bool lat_fits = A.nchain <= 8 && A.chain_rows <= 32;  // four solver warps hold every chain (nx <= 5)
  int modes = thr_modes_per_sm(A, precision, num_sms);
  // one-warp norms, and many modes of models that do not fit the latency kernel, need the throughput kernel
  if (modes == 1 && (nw == 1 || (!lat_fits && A.nitems > 7 * num_sms))) modes = 2;
  // throughput kernel: blocks left open, chains that fit a warp; one-warp modes only where the width was
  // left open too (asked for, they keep their own kernel)
  // (two-warp modes asked for: 5,000 of n = 133 take 134 ms in their own kernel and 105 here, of n = 188 119 and 128)
  const bool thr = open_blocks && modes > 1 && A.chain_rows <= 32 && (warps_per_mode <= 0 || (nw == 2 && A.model_n <= 160) || nw == 4);
  if (blocks_per_sm <= 0 && nw == 4) blocks_per_sm = A.nitems <= 8 * num_sms || (modes == 1 && lat_fits) ? 1 : 2;
  if (nw == 8) blocks_per_sm = 1;  // eight-warp groups: one mode per SM
  const bool lat = !thr && nw == 4 && blocks_per_sm == 1 && lat_fits;  // latency kernel: one mode per SM
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
