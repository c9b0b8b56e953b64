// Precision and group-size dispatch of the perturbation kernel (sbz_pt_impl.cuh).
#include "sbz_pt.cuh"

namespace sbz {

int pt_launch_f32_w1(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_f32_w2_w4(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_f64_w1(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_f64_w2_w4(const PtArgs& A, int nw, int warps_per_block, int blocks_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_lat_f32(const PtArgs& A, int num_sms, cudaStream_t stream);
int pt_launch_lat_f64(const PtArgs& A, int num_sms, cudaStream_t stream);
int pt_launch_thr_f32(const PtArgs& A, int warps, int modes_per_sm, int num_sms, cudaStream_t stream);
int pt_launch_thr_f64(const PtArgs& A, int warps, int modes_per_sm, int num_sms, cudaStream_t stream);
int pt_thr2_resident_f32(int n);
int pt_thr2_resident_f64(int n);

// Warps per mode when the caller leaves it open.  The results of a mode depend on it (order of the norms'
// sums, refinement default).  In mixed precision they do not depend on the kernel that runs it; in all-FP64 the
// latency and throughput kernels form reciprocals of pivots (lat_rcp) where the generic kernel divides.
static int auto_warps_per_mode(int nitems, int num_sms) { return nitems <= 32 * num_sms ? 4 : 1; }

// Modes that share an SM when the caller leaves it open, 1: the latency kernel; warps that run each.  With few modes per
// SM to go round, each gets an SM's FP64 pipes to itself, with many they share them: a mode then takes `slow` times as
// long, but `modes` of them run at once.  A launch lasts about as long as the slower of its longest mode and its
// work over the SMs, slow · max(1, r / modes) in units of the longest mode alone on an SM, with
// r = Σ steps / (longest's steps · SMs).  The choices are one to four modes of four warps, and eight of two or, where
// shared memory holds one block of four only (mixed above 167 equations, all-FP64 above 107), four of two.  The
// table holds measured times (ms, k up to 0.2 h/Mpc) with the SMs full over the longest mode's time alone: mixed n = 47
// 38, 56, 61, 72, 107; n = 82 38.5, 56, 62, 77, 142; n = 98 41, 61, 69, 86, 146; n = 118 42, 63, 71, 91, 142; n = 133
// 46, 79, 90, 106, 171; n = 155 46, 80, 90, 108, 171; n = 182 46.5, 82, 95, 116, 136 (four of two warps).  FP64 n = 38 54, 71,
// 81, 100, 155; n = 82 53, 78, 101, 125, 212; n = 98 60, 88, 115, 139, 219; n = 118 63, 93, 120, 149, 140; n = 133 70, 104,
// 131, 160, 148; n = 182 72, 110, 142, 168, 160 (the last three four of two warps, which all-FP64 runs as fast as four of four).
// The lines follow the rows per lane (above 128 equations two of four warps).  On 120 launches of n = 82 to 182, 456 to
// 4,560 modes, k up to 0.05 and 0.2 h/Mpc, both precisions, this choice is within 4 % of the best of the five shapes, but
// for mixed n > 128 at r = 1.7 (one mode per SM chosen, two 13 to 16 % faster).  Lines on the mode count alone gave up to
// 40 % away where the modes' lengths are close.
struct Sharing { int modes, warps; };
static int plan_items(const PtArgs& A) { return A.plan > 0 ? A.plan : A.nitems; }
static Sharing modes_per_sm(const PtArgs& A, int precision, int num_sms) {
  const bool mixed = precision == SBZ_MIXED;
  static const float mixed_slow[3][4] = {{1.45f, 1.56f, 1.87f, 2.8f}, {1.46f, 1.65f, 2.07f, 3.7f}, {1.75f, 1.97f, 2.33f, 3.75f}};
  static const float fp64_slow[2][4] = {{1.32f, 1.51f, 1.85f, 2.9f}, {1.47f, 1.89f, 2.35f, 3.9f}};
  const int n = A.model_n;
  const float* slow = mixed ? mixed_slow[n <= 64 ? 0 : n <= 128 ? 1 : 2] : fp64_slow[n <= 64 ? 0 : 1];
  const int two = mixed ? pt_thr2_resident_f32(n) : pt_thr2_resident_f64(n);  // modes of two warps
  const Sharing shape[4] = {{2, 4}, {3, 4}, {4, 4}, {two, 2}};
  const double r = (A.load > 0 ? A.load : 0.25 * plan_items(A)) / num_sms;  // modes on the device only: as of a geometric grid up to 0.2 h/Mpc
  Sharing best{1, 4};
  double tb = r > 1 ? r : 1;
  for (int i = 0; i < 4; ++i) {
    const double s = i == 3 && two == 4 ? (mixed ? 2.95 : 2.2) : slow[i];
    const double t = s * (r > shape[i].modes ? r / shape[i].modes : 1);
    if (t < 0.99 * tb) { best = shape[i]; tb = t; }
  }
  return best;
}

PtShape pt_shape(const PtArgs& A, int precision, int warps_per_mode, int blocks_per_sm, int num_sms) {
  const int items = plan_items(A);
  const int nw = warps_per_mode > 0 ? warps_per_mode : auto_warps_per_mode(items, num_sms);
  const bool lat_fits = A.nchain <= 8 && A.chain_rows <= 32;  // four solver warps hold every chain (nx <= 5)
  Sharing sh = modes_per_sm(A, precision, num_sms);
  // one-warp norms, and many modes of models that do not fit the latency kernel, need the throughput kernel
  if (sh.modes == 1 && (nw == 1 || (!lat_fits && items > 7 * num_sms))) sh.modes = 2;
  // throughput kernel: blocks left open, chains that fit a warp; one-warp modes only where the width was
  // left open too (asked for, they keep their own kernel)
  // (two-warp modes asked for: 5,000 of n = 133 take 134 ms in their own kernel and 105 here, of n = 188 119 and 128)
  if (blocks_per_sm <= 0 && sh.modes > 1 && A.chain_rows <= 32 && (warps_per_mode <= 0 || (nw == 2 && A.model_n <= 160) || nw == 4))
    return PtShape{PT_THROUGHPUT, nw, sh.warps, sh.modes, 0};
  if (blocks_per_sm <= 0 && nw == 4) blocks_per_sm = items <= 8 * num_sms || (sh.modes == 1 && lat_fits) ? 1 : 2;
  if (nw == 8) blocks_per_sm = 1;  // eight-warp groups: one mode per SM
  if (nw == 4 && blocks_per_sm == 1 && lat_fits) return PtShape{PT_LATENCY, nw, nw, 1, 1};  // one mode per SM
  return PtShape{PT_GENERIC, nw, nw, 0, blocks_per_sm};
}

int pt_launch(const PtArgs& A, int precision, int warps_per_block, int warps_per_mode, int blocks_per_sm, int num_sms,
              cudaStream_t stream) {
  if (warps_per_block <= 0) warps_per_block = 4;
  const PtShape s = pt_shape(A, precision, warps_per_mode, blocks_per_sm, num_sms);
  const int nw = s.nw;
  if (nw != 1 && nw != 2 && nw != 4 && nw != 8) return SBZ_ERR_ARG;
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
    if (s.kernel == PT_THROUGHPUT) return pt_launch_thr_f32(B, s.warps, s.modes, num_sms, stream);
    if (s.kernel == PT_LATENCY) return pt_launch_lat_f32(B, num_sms, stream);
    return nw == 1 ? pt_launch_f32_w1(B, nw, warps_per_block, s.blocks, num_sms, stream)
                   : pt_launch_f32_w2_w4(B, nw, warps_per_block, s.blocks, num_sms, stream);
  }
  PtArgs B = A;
  B.norm_warps = nw;
  if (s.kernel == PT_THROUGHPUT) return pt_launch_thr_f64(B, s.warps, s.modes, num_sms, stream);
  if (s.kernel == PT_LATENCY) return pt_launch_lat_f64(A, num_sms, stream);
  return nw == 1 ? pt_launch_f64_w1(A, nw, warps_per_block, s.blocks, num_sms, stream) : pt_launch_f64_w2_w4(A, nw, warps_per_block, s.blocks, num_sms, stream);
}

}  // namespace sbz
