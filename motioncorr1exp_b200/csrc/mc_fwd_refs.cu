// Forward row pass of libmc for two-level lengths with dark/gain references
// (sm_100a; DFAlign.cu:710-806).
#include <algorithm>

#include "kcommon.cuh"

namespace mc {

// Forward rows with dark/gain references: two teams of T threads side by
// side, each one packed transform -- two image rows, or one row with its two
// reference sets (two_outputs).  Step A's loads decode the pixel and apply the
// references straight from global memory, N2 independent loads of each array a
// thread, and Z goes back into the exchange buffer: 29.7 KB per transform where
// staged rows and a second buffer took 59 (n = 3710), and no pass of one
// element a thread and trip between the loads and the transform.  The CTA then
// writes its rows' half spectra: four rows as one 32-byte sector per kx, or two
// rows as 16 bytes in each set.  Measured, 16 frames of 3710^2 uint16 with dark
// and gain: 5.63 -> 2.55 ms.
template <int N1, int N2, typename Px>
__global__ void __launch_bounds__(2 * TwoLevel<N1, N2>::T, tl_min_blocks(TwoLevel<N1, N2>::T) / 2) k_fwd_rows2l_refs(FwdRowsArgs a) {
  using TL = TwoLevel<N1, N2>;
  constexpr int N = TL::N, T = TL::T;
  extern __shared__ float2 dynref[];
  const int tid = threadIdx.x, team = tid / T, lt = tid - team * T;
  float2* ysm = dynref + (size_t)team * N;
  const Px* f = reinterpret_cast<const Px*>(fwd_frame(a));
  float2* outA = a.outA + blockIdx.y * a.out_stride;
  // the dark and gain of the packed sequence's halves (null: 0 and 1)
  const bool two_sets = a.two_outputs != 0;
  const int rows = two_sets ? 1 : 2;
  const int y0 = 2 * rows * blockIdx.x;               // the CTA's first row
  const bool both = two_sets || y0 + 2 < a.nu;        // the second team has rows of its own
  const long long r0 = (long long)(a.offy + y0 + (both ? team * rows : 0)) * a.nx + a.offx;
  const long long r1 = two_sets ? r0 : r0 + a.nx;
  const float *d0 = a.dark, *d1 = two_sets ? a.dark2 : a.dark;
  const float *g0 = a.norm, *g1 = two_sets ? a.norm2 : a.norm;
  TL::template run<false, true, kFwdRowsPaired>(
      ysm, a.tw + N,
      [&](int x) {
        const float p0 = (float)f[r0 + x], p1 = two_sets ? p0 : (float)f[r1 + x];
        const float b0 = d0 ? __ldg(d0 + r0 + x) : 0.f, b1 = d1 ? __ldg(d1 + r1 + x) : 0.f;
        const float m0 = g0 ? __ldg(g0 + r0 + x) : 1.f, m1 = g1 ? __ldg(g1 + r1 + x) : 1.f;
        // hbuf, hbuf2 (DFAlign.cu:724-725), rounded before the transform's sums
        return make_float2(__fmul_rn(p0 - b0, m0), __fmul_rn(p1 - b1, m1));
      },
      [&](int k, float2 v) { ysm[k] = v; }, (N1 - 1) / 2, lt);
  __syncthreads();
  // X = (Z(k) + conj Z(-k))/2, Y = -i (Z(k) - conj Z(-k))/2
  auto even = [&](const float2* z, int k) {
    const float2 u = z[k], v = z[k == 0 ? 0 : N - k];
    return make_float2(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
  };
  auto odd = [&](const float2* z, int k) {
    const float2 u = z[k], v = z[k == 0 ? 0 : N - k];
    return make_float2(0.5f * (u.y + v.y), -0.5f * (u.x - v.x));
  };
  for (int i = tid; i < 2 * a.hk; i += 2 * T) {
    const int k = i >> 1, h = i & 1;
    if (two_sets) {
      // set h of rows y0, y0 + 1
      float2* o = h ? a.outB + blockIdx.y * a.out_stride : outA;
      const float2 u = h ? odd(dynref, k) : even(dynref, k), v = h ? odd(dynref + N, k) : even(dynref + N, k);
      *reinterpret_cast<float4*>(o + (long long)k * a.ldt + y0) = make_float4(u.x, u.y, v.x, v.y);
    } else if (h == 0 || both) {
      const float2* z = dynref + (size_t)h * N;
      const float2 u = even(z, k), v = odd(z, k);
      *reinterpret_cast<float4*>(outA + (long long)k * a.ldt + y0 + 2 * h) = make_float4(u.x, u.y, v.x, v.y);
    }
  }
}

template <int A, int B, typename PX>
cudaError_t launch_refs_rows(const FwdRowsArgs& a, cudaStream_t st) {
  const size_t smem = 2 * (size_t)A * B * sizeof(float2);
  cudaError_t e = allow_smem((const void*)k_fwd_rows2l_refs<A, B, PX>, smem);
  if (e != cudaSuccess) return e;
  const int rows = a.two_outputs ? 2 : 4;
  k_fwd_rows2l_refs<A, B, PX><<<dim3((a.nu + rows - 1) / rows, std::max(a.nfr, 1)), 2 * TwoLevel<A, B>::T, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fwd_rows2l_refs(const FwdRowsArgs& a, cudaStream_t st) {
  int n1 = 0, n2 = 0;
  if (!two_level_split(a.nu, n1, n2)) return cudaErrorInvalidValue;
#define MC_REFS_LAUNCH(A, B)                                             \
  if (n1 == (A) && n2 == (B)) {                                          \
    switch (a.mode) {                                                    \
      case 0: return launch_refs_rows<A, B, int8_t>(a, st);              \
      case MC_MODE_U8: return launch_refs_rows<A, B, uint8_t>(a, st);    \
      case 1: return launch_refs_rows<A, B, int16_t>(a, st);             \
      case 6: return launch_refs_rows<A, B, uint16_t>(a, st);            \
      case MC_MODE_F16: return launch_refs_rows<A, B, __half>(a, st);    \
      default: return launch_refs_rows<A, B, float>(a, st);              \
    }                                                                    \
  }
  MC_TWO_LEVEL_LIST(MC_REFS_LAUNCH)
#undef MC_REFS_LAUNCH
  return cudaErrorInvalidValue;
}

}  // namespace mc
