// Hand-written sm_100a kernels of the drift-correction path, in translation
// units that compile in parallel:
//   mc_fwd.cu, mc_fwd_raw.cu, mc_fwd_refs.cu, mc_fwd_dif.cu   k_fwd_rows*,
//        k_rows_fft*: decode + dark/gain + crop + row R2C with transposed store
//        (DFAlign.cu:710-806), column FFT with Fourier-crop binning
//        (cufunc.cu:162-176, 223-227)
//   mc_pair.cu, mc_pair_cols.cu   k_pair_cols*, k_pair_rows*: cross power x
//        B-factor + pruned inverse FFTs onto the pbx window (cufunc.cu:229-233,
//        343-407)
//   mc_sum.cu    k_peak, k_ramp, k_shift_acc, k_sum_cols*, k_c2r_rows*,
//        k_count_sum, k_objective* (cufunc.cu:372-497, DFAlign.cu:1287-1292)
//   mc_solve.cu  k_solve, k_solve_smem: drift solve (DFAlign.cu:914-948, 1056-1139)
//   this file    host helpers shared by all of them
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include "kernels.cuh"

namespace mc {

// Raise-only, thread-safe opt-in to large dynamic shared memory.  The
// attribute is per function and per device; two host threads that launch
// the same kernel with different sizes must never lower it under each other.
cudaError_t allow_smem(const void* func, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  size_t& cur = done[{dev, func}];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

// Chosen by a model of one CTA's time: every stage runs ceil(butterflies /
// threads) rounds, each costing a fixed latency plus its radix' traffic and
// arithmetic, so thread counts that leave the last round of a stage nearly
// empty lose; CTAs per SM follow from threads (80 registers each) and shared
// memory.  The best is the one that finishes most transforms per SM and time.
MixedShape mixed_shape(const FftPlan1D& p, int count, bool gather) {
  MixedShape best{1, 256, (size_t)2 * p.n * sizeof(float2)};
  double top = -1.0;
  for (int B = 1; B <= 16 && (B == 1 || B <= count); B *= 2) {
    const size_t smem = (size_t)2 * B * p.n * sizeof(float2);
    if (smem > 200 * 1024 && B > 1) break;
    for (int th = 64; th <= kMixedMaxThreads; th += 32) {
      const double res = std::min({2048 / th, 65536 / (th * 80), (int)(227 * 1024 / (smem + 1024)), 32});
      if (res < 1) continue;
      double t = 40.0;
      for (int s = 0; s < p.nst; s++) {
        const FftStage& st = p.st[s];
        const int nq = p.n / st.R, items = nq * B;
        auto rounds = [&](int k) { return (double)((k + th - 1) / th); };
        if (st.kind == kStageSymmetric) {
          const int h = (st.R - 1) / 2, ng = (h + kPrimePairs - 1) / kPrimePairs;
          t += 40.0 + rounds(items * (h + 1)) * 24.0 + rounds(items * ng) * (20.0 + h * 16.0);
        } else if (st.kind == kStageDirect) {
          t += 40.0 + rounds(items * st.R) * 12.0 + rounds(items * ((st.R + 7) / 8)) * (20.0 + st.R * 28.0);
        } else if (st.kind == kStageGeneric) {
          t += 40.0 + rounds(items * st.R) * (20.0 + 8.0 * st.R);
        } else {
          t += 40.0 + rounds(items) * (30.0 + 8.0 * st.R);
        }
      }
      // CTAs that run at once do not finish sooner than one of them
      double rate = 1.0 / (std::max(1.0, (double)count / (148.0 * res * B)) * t);
      if (gather && B >= 2) rate *= 1.2;
      if (rate > top) {
        top = rate;
        best = {B, th, smem};
      }
    }
  }
  return best;
}

}  // namespace mc
