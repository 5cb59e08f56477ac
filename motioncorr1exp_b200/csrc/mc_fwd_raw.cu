// Forward row pass of libmc for two-level lengths without dark/gain references
// (sm_100a): two rows packed as one complex FFT (DFAlign.cu:710-806).
#include <algorithm>

#include "kcommon.cuh"

namespace mc {

// Forward rows without references, four rows per CTA: two teams of T threads
// each run one packed two-row transform, its step-A loads decoding the pixels
// straight from global memory (N2 independent loads of either row a thread;
// staging the raw rows first cost the CTA a phase of its own and shared memory
// for another CTA: 40 x 3710^2 uint8 2.61 -> 2.10 ms, 24 x 4096^2 float 2.02 ->
// 1.20, 16 x 1024^2 float 73 -> 61 us); they write their spectrum Z back into
// their exchange buffer after the barrier that follows the step-B reads; then
// the CTA writes the four rows' half spectra as one 32-byte sector per kx (two
// threads per sector) instead of two half sectors from two CTAs.  The last
// CTA of an odd pair count runs its second team on a copy of the first pair
// and stores only the first.
template <int N1, int N2, typename Px, bool PAIRED>
__global__ void __launch_bounds__(2 * TwoLevel<N1, N2>::T, tl_min_blocks(TwoLevel<N1, N2>::T) / 2) k_fwd_rows2l_raw4(FwdRowsArgs a) {
  using TL = TwoLevel<N1, N2>;
  constexpr int N = TL::N, T = TL::T;
  extern __shared__ float2 dynraw[];
  const int tid = threadIdx.x, team = tid / T, lt = tid - team * T;
  float2* ysm = dynraw + (size_t)team * N;
  const int y0 = 4 * blockIdx.x;
  float2* outA = a.outA + blockIdx.y * a.out_stride;
  const bool two = y0 + 2 < a.nu;  // the second row pair exists
  const Px* f = reinterpret_cast<const Px*>(fwd_frame(a));
  auto row = [&](int j) { return f + (long long)(a.offy + y0 + (two ? j : (j & 1))) * a.nx + a.offx; };
  const Px *p0 = row(2 * team), *p1 = row(2 * team + 1);
  TL::template run<false, true, PAIRED>(
      ysm, a.tw + N, [&](int x) { return make_float2((float)p0[x], (float)p1[x]); },
      [&](int k, float2 v) { ysm[k] = v; }, (N1 - 1) / 2, lt);
  __syncthreads();
  const int nh = two ? 2 : 1;
  for (int i = tid; i < 2 * a.hk; i += 2 * T) {
    const int k = i >> 1, h = i & 1;
    if (h < nh) {
      const float2* zs = dynraw + (size_t)h * N;
      const float2 z = zs[k];
      const float2 zc = zs[k == 0 ? 0 : N - k];
      const float2 X = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
      const float2 Y = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
      *reinterpret_cast<float4*>(outA + (long long)k * a.ldt + y0 + 2 * h) = make_float4(X.x, X.y, Y.x, Y.y);
    }
  }
}

template <int A, int B, typename PX, bool PR>
cudaError_t launch_raw_rows_p(const FwdRowsArgs& a, int grid, cudaStream_t st) {
  const size_t smem = 2 * (size_t)A * B * sizeof(float2);
  cudaError_t e = allow_smem((const void*)k_fwd_rows2l_raw4<A, B, PX, PR>, smem);
  if (e != cudaSuccess) return e;
  k_fwd_rows2l_raw4<A, B, PX, PR><<<dim3((grid + 1) / 2, std::max(a.nfr, 1)), 2 * TwoLevel<A, B>::T, smem, st>>>(a);
  return cudaGetLastError();
}

// Raw-row launch with the radix-53 pairing the schedule asks for (other
// lengths have no radix-53 step: one instantiation)
template <int A, int B, typename PX>
cudaError_t launch_raw_rows(const FwdRowsArgs& a, bool paired, int grid, cudaStream_t st) {
  if constexpr (A == 53) {
    if (paired != kFwdRowsPaired) return launch_raw_rows_p<A, B, PX, !kFwdRowsPaired>(a, grid, st);
  }
  return launch_raw_rows_p<A, B, PX, kFwdRowsPaired>(a, grid, st);
}

cudaError_t launch_fwd_rows2l_refs(const FwdRowsArgs& a, cudaStream_t st);

cudaError_t launch_fwd_rows2l(const FwdRowsArgs& a, cudaStream_t st) {
  int n1 = 0, n2 = 0;
  if (!two_level_split(a.nu, n1, n2)) return cudaErrorInvalidValue;
  const int grid = a.two_outputs ? a.nu : a.nu / 2;
  const bool raw = !a.two_outputs && !a.dark && !a.dark2 && !a.norm && !a.norm2;
  // the pairing of the radix-53 step (only N1 = 53 has one): schedule or built-in
  const bool paired = a.paired == 0 ? kFwdRowsPaired : a.paired == 2;
#define MC_TL_RAW(A, B, PX) return launch_raw_rows<A, B, PX>(a, paired, grid, st);
#define MC_TL_LAUNCH(A, B)                                                                           \
  if (n1 == (A) && n2 == (B)) {                                                                      \
    if (raw) {                                                                                       \
      switch (a.mode) {                                                                              \
        case 0: MC_TL_RAW(A, B, int8_t)                                                              \
        case MC_MODE_U8: MC_TL_RAW(A, B, uint8_t)                                                    \
        case 1: MC_TL_RAW(A, B, int16_t)                                                             \
        case 6: MC_TL_RAW(A, B, uint16_t)                                                            \
        case MC_MODE_F16: MC_TL_RAW(A, B, __half)                                                    \
        default: MC_TL_RAW(A, B, float)                                                              \
      }                                                                                              \
    }                                                                                                \
    return launch_fwd_rows2l_refs(a, st);                                                            \
  }
  MC_TWO_LEVEL_LIST(MC_TL_LAUNCH)
#undef MC_TL_LAUNCH
#undef MC_TL_RAW
  return cudaErrorInvalidValue;
}

}  // namespace mc
