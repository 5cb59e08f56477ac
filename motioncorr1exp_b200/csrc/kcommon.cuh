// Device code shared by the kernel translation units of libmc (mc_fwd*.cu,
// mc_pair*.cu, mc_sum.cu): constants, the two-level register FFT and the raw-row
// staging helpers.
#pragma once
#include <cuda_fp16.h>
#include <math.h>
#include <stdint.h>

#include "kernels.cuh"
#include "codelets_gen.cuh"
#include "mixed_fft.cuh"

namespace mc {

namespace {

constexpr int kThreads = 256;

}  // namespace

// Frame read by a forward CTA (direct pointer, or the run's base from the
// device-side slot plus the first frame's offset; frame blockIdx.y of the launch).
__device__ __forceinline__ const void* fwd_frame(const FwdRowsArgs& a) {
  const char* f = a.frames_slot ? static_cast<const char*>(*a.frames_slot) + a.frame_offset
                                : static_cast<const char*>(a.frame);
  return f + (long long)blockIdx.y * a.frame_stride;
}

// ================================================== two-level transforms ==
// Length N = N1*N2 with n = n1 + N1*n2 and k = k2 + N2*k1:
//   Y[n1][k2]      = W_N^(n1 k2) * sum_n2 x[n1 + N1 n2] W_N2^(n2 k2)   thread n1: N2-point codelet
//   X[k2 + N2 k1]  = sum_n1 Y[n1][k2] W_N1^(n1 k1)                    thread k2: N1-point codelet
// so a whole transform costs one shared-memory exchange.  N1 = 53 uses the
// generated radix-53 butterfly.  One CTA (a team of `T2L` threads) per
// transform; step A's factors W_N^(n1 k2) come from a global table laid out
// [k2][n1] (fft_tables), so the threads n1 of a warp read consecutive words.
// Built-in radix-53 schedules of the forward row / column transforms: two
// output pairs per loop pass in both (measured on c2: the row pass 9 %
// faster paired; the column pass 12 % faster paired once its stores lost
// the crop test and the scale, 27 % slower before); a schedule
// (mc_schedule_set, the autotuner) can pick either.
constexpr bool kFwdRowsPaired = true;
constexpr bool kFwdColsPaired = true;
// Resident CTAs per SM the two-level transforms of T threads are compiled for
// (register cap): 168 registers at 96 and 64 threads, 128 at 32.  4096^2 column
// pass, 24 frames, with four / five / six CTAs of 64 threads 1062, 940, 942 us,
// 2048^2 row pass 311, 310, 263; 16 x 1024^2 row pass with 4 / 10 / 16 CTAs of 32
// 66, 65, 61; 96 threads with five (136 registers, spills): 3710^2 column pass
// 1.67 -> 2.14 ms.
constexpr int tl_min_blocks(int T) { return T == 96 ? 4 : T == 64 ? 6 : 16; }

template <int N1, int N2>
struct TwoLevel {
  static constexpr int N = N1 * N2;
  static constexpr int T = ((N1 > N2 ? N1 : N2) + 31) / 32 * 32;

  // step A + exchange + step B; load(i) gives x[i], store(k, X[k]) takes the
  // result; tw[k2 * N1 + n1] = exp(-2 pi i n1 k2 / N).  For N1 = 53 only the
  // outputs with k1 or N1 - k1 <= kmax are formed (pruned transforms).
  // T >= N2, so each thread owns at most one k2 in step B; with
  // SYNC_STORE a barrier follows every thread's step-B reads of ysm, which
  // lets store() write back into ysm.
  template <bool INV, bool SYNC_STORE, bool PAIRED = false, class Load, class Store>
  __device__ static void run(float2* ysm, const float2* __restrict__ tw, Load&& load, Store&& store,
                             int kmax = (N1 - 1) / 2, int lt_team = -1) {
    static_assert(T >= N2, "one k2 per thread");
    // lt_team: the thread's index in its team of T when a CTA runs several
    // transforms side by side (every team takes the same barriers)
    const int lt = lt_team >= 0 ? lt_team : (int)threadIdx.x;
    if (lt < N1) {
      float2 x[N2];
#pragma unroll
      for (int n2 = 0; n2 < N2; n2++) x[n2] = load(lt + N1 * n2);
      fft_reg<N2, INV>(x);
#pragma unroll
      for (int k2 = 0; k2 < N2; k2++) {
        float2 w = __ldg(tw + k2 * N1 + lt);
        if (INV) w.y = -w.y;
        ysm[k2 * N1 + lt] = k2 ? cmul(x[k2], w) : x[k2];
      }
    }
    __syncthreads();
    const bool act = lt < N2;
    float2 v[N1];
    if (act) {
#pragma unroll
      for (int n1 = 0; n1 < N1; n1++) v[n1] = ysm[lt * N1 + n1];
    }
    if (SYNC_STORE) __syncthreads();
    if constexpr (N1 == 53) {
      // compact radix-53 DFT: small code, outputs stored as they are formed
      if (act) dft_r53_compact<INV, PAIRED>(v, [&](int k1, float2 x) { store(lt + N2 * k1, x); }, kmax);
    } else {
      if (act) fft_reg<N1, INV>(v);
      if (act) {
#pragma unroll
        for (int k1 = 0; k1 < N1; k1++) store(lt + N2 * k1, v[k1]);
      }
    }
  }
};

// Stage the two packed input rows of one transform of k_fwd_rows in shared
// memory: every thread of the CTA issues independent typed loads of the raw
// pixels.
template <typename Px>
__device__ __forceinline__ void stage_rows(float2* xin, const FwdRowsArgs& a, long long r0, long long r1, int n,
                                           int nth) {
  const Px* f = reinterpret_cast<const Px*>(fwd_frame(a));
  const bool hasd = a.dark != nullptr, hasn = a.norm != nullptr;
  if (a.two_outputs) {
#pragma unroll 4
    for (int x = threadIdx.x; x < n; x += nth) {
      const long long i0 = r0 + x;
      const float raw = (float)f[i0];
      const float d1 = hasd ? a.dark[i0] : 0.f;
      const float d2 = hasd ? (a.dark2 ? a.dark2[i0] : 0.f) : 0.f;
      const float g1 = hasn ? a.norm[i0] : 1.f;
      const float g2 = hasn ? (a.norm2 ? a.norm2[i0] : 1.f) : 1.f;
      xin[x] = make_float2((raw - d1) * g1, (raw - d2) * g2);  // hbuf, hbuf2 (DFAlign.cu:724-725)
    }
  } else if (hasd || hasn) {
#pragma unroll 4
    for (int x = threadIdx.x; x < n; x += nth) {
      const long long i0 = r0 + x, i1 = r1 + x;
      const float re = ((float)f[i0] - (hasd ? a.dark[i0] : 0.f)) * (hasn ? a.norm[i0] : 1.f);
      const float im = ((float)f[i1] - (hasd ? a.dark[i1] : 0.f)) * (hasn ? a.norm[i1] : 1.f);
      xin[x] = make_float2(re, im);
    }
  } else {
#pragma unroll 8
    for (int x = threadIdx.x; x < n; x += nth) xin[x] = make_float2((float)f[r0 + x], (float)f[r1 + x]);
  }
}

// Raw pixels of one crop row into shared memory with aligned 16-byte loads:
// the bytes of [src, src + n) land at dst[d + i] with d = src mod 16, so
// every interior 16-byte chunk keeps its alignment in shared memory; the
// unaligned head and tail go pixel by pixel.  Every load stays inside the row.
template <typename Px>
__device__ __forceinline__ void stage_raw_row(unsigned char* dst, const Px* src, int n, int tid, int nth) {
  const uintptr_t s = reinterpret_cast<uintptr_t>(src);
  const uintptr_t e = s + (uintptr_t)n * sizeof(Px);
  const uintptr_t a0 = s & ~(uintptr_t)15;
  uintptr_t as = (s + 15) & ~(uintptr_t)15;
  uintptr_t ae = e & ~(uintptr_t)15;
  if (as > ae) as = ae = e;  // row shorter than one aligned chunk: all pixel by pixel
  const int head = (int)((as - s) / sizeof(Px)), tail0 = (int)((ae - s) / sizeof(Px));
  Px* dpx = reinterpret_cast<Px*>(dst + (s - a0));
  for (int i = tid; i < head; i += nth) dpx[i] = src[i];
  for (int i = tail0 + tid; i < n; i += nth) dpx[i] = src[i];
  const int chunks = (int)((ae - as) / 16);
  const uint4* g = reinterpret_cast<const uint4*>(as);
  uint4* d4 = reinterpret_cast<uint4*>(dst + (as - a0));
  for (int c = tid; c < chunks; c += nth) d4[c] = __ldg(g + c);
}

// Two-level splits compiled in (N1, N2).
#define MC_TWO_LEVEL_LIST(X) X(53, 70) X(64, 64) X(32, 64) X(32, 32) X(16, 16) X(16, 32)
bool two_level_split(int n, int& n1, int& n2);

}  // namespace mc
