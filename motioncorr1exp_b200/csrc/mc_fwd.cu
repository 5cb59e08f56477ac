// Forward transforms of libmc (sm_100a): decode + dark/gain + crop + row FFT
// with transposed store (DFAlign.cu:710-806, general form), the column FFT with
// Fourier-crop binning (cufunc.cu:162-176, 223-227) and the batched row
// transforms of the inverse passes.  The two-level row kernels live in
// mc_fwd_raw.cu, the radix-2 split forms for lengths 2N in mc_fwd_dif.cu.
#include <algorithm>

#include "kcommon.cuh"

namespace mc {

// =========================================================== forward rows ==
// The packed input rows of B transforms (row pairs q0 .. q0 + nb - 1, zero
// beyond) into xin.  Pixels of one or two bytes without references first land
// as raw rows in `scratch` (the engine's other buffer) by aligned 16-byte
// loads and are decoded from there: a pixel at a time from global memory, the
// few loads a thread keeps in flight set the pace (row pass per frame 205 ->
// 182 us at 4092^2 uint8, 15.7 -> 13.5 at 1500^2 half, 2.2 / 2.2 at 520^2 int16).
template <typename Px>
__device__ __forceinline__ void stage_pairs(float2* scratch, float2* xin, const FwdRowsArgs& a, int q0, int nb, int B,
                                            bool raw) {
  const int nu = a.nu, tid = threadIdx.x, nth = blockDim.x;
  const int rb = (nu * (int)sizeof(Px) + 30) / 16 * 16;  // a staged row, any alignment
  auto row = [&](int y) { return (long long)(a.offy + y) * a.nx + a.offx; };
  if (sizeof(Px) < 4 && raw && 2 * rb <= nu * (int)sizeof(float2)) {
    unsigned char* rows = reinterpret_cast<unsigned char*>(scratch);
    const Px* f = reinterpret_cast<const Px*>(fwd_frame(a));
    // short rows: a group of warps each, all in flight together
    const int ng = min(nth / 32, 2 * nb), gth = nth / 32 / ng * 32, grp = tid / gth;
    if (grp < ng)
      for (int i = grp; i < 2 * nb; i += ng)
        stage_raw_row<Px>(rows + i * rb, f + row(2 * q0 + i), nu, tid - grp * gth, gth);
    __syncthreads();
    for (int b = 0; b < B; b++) {
      float2* x = xin + (size_t)b * nu;
      if (b >= nb) {
        for (int i = tid; i < nu; i += nth) x[i] = make_float2(0.f, 0.f);
        continue;
      }
      auto staged = [&](int i) {
        return reinterpret_cast<const Px*>(rows + i * rb + (reinterpret_cast<uintptr_t>(f + row(2 * q0 + i)) & 15));
      };
      const Px *p0 = staged(2 * b), *p1 = staged(2 * b + 1);
#pragma unroll 4
      for (int i = tid; i < nu; i += nth) x[i] = make_float2((float)p0[i], (float)p1[i]);
    }
    return;
  }
  for (int b = 0; b < B; b++) {
    float2* x = xin + (size_t)b * nu;
    if (b >= nb) {
      for (int i = tid; i < nu; i += nth) x[i] = make_float2(0.f, 0.f);
      continue;
    }
    const int y0 = a.two_outputs ? q0 + b : 2 * (q0 + b);
    stage_rows<Px>(x, a, row(y0), a.two_outputs ? row(y0) : row(y0 + 1), nu, nth);
  }
}

// Lengths without a compiled split: B packed transforms (two rows each, or
// the two reference sets of one row) per CTA on the mixed-radix engine.  With
// B >= 2 the CTA's half spectra of one kx fill 32-byte sectors of the
// transposed store.
__global__ void __launch_bounds__(kMixedMaxThreads, kMixedMinBlocks) k_fwd_rows(FwdRowsArgs a, int B) {
  extern __shared__ float2 sm[];
  const int nu = a.nu;
  float2* s0 = sm;
  float2* s1 = sm + (size_t)B * nu;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int q0 = blockIdx.x * B, npair = a.two_outputs ? nu : nu / 2;
  const int nb = min(B, npair - q0);
  const bool raw = !a.two_outputs && !a.dark && !a.norm;
  switch (a.mode) {
    case 0: stage_pairs<int8_t>(s0, s1, a, q0, nb, B, raw); break;
    case MC_MODE_U8: stage_pairs<uint8_t>(s0, s1, a, q0, nb, B, raw); break;
    case 1: stage_pairs<int16_t>(s0, s1, a, q0, nb, B, raw); break;
    case 6: stage_pairs<uint16_t>(s0, s1, a, q0, nb, B, raw); break;
    case MC_MODE_F16: stage_pairs<__half>(s0, s1, a, q0, nb, B, raw); break;
    default: stage_pairs<float>(s0, s1, a, q0, nb, B, raw); break;
  }
  __syncthreads();
  fft_exec<false, false>(
      s0, s1, a.plan, B, nu, a.tw, tid, nth, [&](int b, int i) { return s1[b * nu + i]; },
      [&](float2* dst, int b, int i, float2 v) { dst[b * nu + i] = v; });
  __syncthreads();
  const float2* Z = (a.plan.nst & 1) ? s0 : s1;
  float2* outA = a.outA + blockIdx.y * a.out_stride;
  float2* outB = a.two_outputs ? a.outB + blockIdx.y * a.out_stride : nullptr;
  // split the two real transforms: X = (Z(k) + conj Z(-k))/2, Y = -i (Z(k) - conj Z(-k))/2
  for (int t = tid; t < a.hk * B; t += nth) {
    const int k = t / B, b = t - k * B;
    if (b >= nb) continue;
    const float2* z0 = Z + b * nu;
    const float2 z = z0[k];
    const float2 zc = z0[k == 0 ? 0 : nu - k];
    const float2 X = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
    const float2 Y = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
    if (a.two_outputs) {
      outA[(long long)k * a.ldt + q0 + b] = X;
      outB[(long long)k * a.ldt + q0 + b] = Y;
    } else {
      *reinterpret_cast<float4*>(outA + (long long)k * a.ldt + 2 * (q0 + b)) = make_float4(X.x, X.y, Y.x, Y.y);
    }
  }
}

bool two_level_split(int n, int& n1, int& n2);
cudaError_t launch_fwd_rows2l(const FwdRowsArgs& a, cudaStream_t st);
cudaError_t launch_rows_fft2l(const RowsFftArgs& a, bool inverse, cudaStream_t st);

cudaError_t launch_fwd_rows_dif(const FwdRowsArgs& a, cudaStream_t st);
cudaError_t launch_rows_fft_dif(const RowsFftArgs& a, cudaStream_t st);
bool dif_supported(int n);

cudaError_t launch_fwd_rows(const FwdRowsArgs& a, cudaStream_t st) {
  int n1, n2;
  if (two_level_split(a.nu, n1, n2)) return launch_fwd_rows2l(a, st);
  const bool raw = !a.two_outputs && !a.dark && !a.dark2 && !a.norm && !a.norm2;
  if (raw && dif_supported(a.nu)) return launch_fwd_rows_dif(a, st);
  const int npair = a.two_outputs ? a.nu : a.nu / 2;
  const MixedShape sh = mixed_shape(a.plan, npair * std::max(a.nfr, 1), true);
  cudaError_t e = allow_smem((const void*)k_fwd_rows, sh.smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((npair + sh.B - 1) / sh.B, std::max(a.nfr, 1));
  k_fwd_rows<<<grid, sh.threads, sh.smem, st>>>(a, sh.B);
  return cudaGetLastError();
}

// ========================================================= row transforms ==
template <bool INV>
__global__ void __launch_bounds__(kMixedMaxThreads, kMixedMinBlocks) k_rows_fft(RowsFftArgs a, int B) {
  extern __shared__ float2 sm[];
  const int n = a.plan.n;
  const int row0 = blockIdx.x * B;
  const int nb = min(B, a.nrows - row0);
  const float2* in = a.in + blockIdx.y * a.in_stride + (long long)row0 * a.ld_in;
  float2* out = a.out + blockIdx.y * a.out_stride + (long long)row0 * a.ld_out;
  const int shift = n - a.n_out;
  // in place: every stage but the last one leaves `out` alone, and a barrier
  // (or, for a single stage, the thread's own order) precedes the last
  fft_exec<INV, false>(
      sm, sm + (size_t)B * n, a.plan, B, n, a.tw, threadIdx.x, blockDim.x,
      [&](int b, int i) { return b < nb ? in[(long long)b * a.ld_in + i] : make_float2(0.f, 0.f); },
      [&](float2*, int b, int i, float2 v) {
        int o = i;
        if (i >= a.keep_lo) {
          if (i < a.keep_lo + shift) return;
          o = i - shift;
        }
        if (b < nb) out[(long long)b * a.ld_out + o] = make_float2(v.x * a.scale, v.y * a.scale);
      });
}

cudaError_t launch_rows_fft(const RowsFftArgs& a, bool inverse, cudaStream_t st) {
  int n1, n2;
  if (two_level_split(a.plan.n, n1, n2)) return launch_rows_fft2l(a, inverse, st);
  if (!inverse && dif_supported(a.plan.n)) return launch_rows_fft_dif(a, st);
  const MixedShape sh = mixed_shape(a.plan, a.nrows * std::max(a.nfr, 1), false);
  const dim3 grid((a.nrows + sh.B - 1) / sh.B, std::max(a.nfr, 1));
  cudaError_t e;
  if (inverse) {
    e = allow_smem((const void*)k_rows_fft<true>, sh.smem);
    if (e != cudaSuccess) return e;
    k_rows_fft<true><<<grid, sh.threads, sh.smem, st>>>(a, sh.B);
  } else {
    e = allow_smem((const void*)k_rows_fft<false>, sh.smem);
    if (e != cudaSuccess) return e;
    k_rows_fft<false><<<grid, sh.threads, sh.smem, st>>>(a, sh.B);
  }
  return cudaGetLastError();
}

// Batched rows: out_row[i] = scale * X[i < keep_lo ? i : i + (n - n_out)].  In
// place when nothing is cropped (a barrier inside the transform separates a
// row's reads from its stores), so the row is read with plain loads: __ldg is
// for memory that the kernel does not write.
template <int N1, int N2, bool INV, bool PAIRED, bool PLAIN = false>
__global__ void __launch_bounds__(TwoLevel<N1, N2>::T, tl_min_blocks(TwoLevel<N1, N2>::T)) k_rows_fft2l(RowsFftArgs a) {
  using TL = TwoLevel<N1, N2>;
  __shared__ float2 ysm[TL::N];
  const long long row = blockIdx.x;
  const float2* in = a.in + blockIdx.y * a.in_stride + row * a.ld_in;
  float2* out = a.out + blockIdx.y * a.out_stride + row * a.ld_out;
  if constexpr (PLAIN) {
    // every output kept, unscaled (the forward column pass without a Fourier
    // crop): no per-output crop test or multiply (2.47 -> 2.15 ms per c2 movie)
    TL::template run<INV, false, PAIRED>(ysm, a.tw + TL::N, [&](int i) { return in[i]; },
                                         [&](int k, float2 v) { out[k] = v; });
  } else {
    const int shift = TL::N - a.n_out, keep = a.keep_lo;
    const float sc = a.scale;
    TL::template run<INV, false, PAIRED>(ysm, a.tw + TL::N, [&](int i) { return in[i]; },
                          [&](int k, float2 v) {
                            int o;
                            if (k < keep) o = k;
                            else if (k >= keep + shift) o = k - shift;
                            else return;
                            out[o] = make_float2(v.x * sc, v.y * sc);
                          });
  }
}


bool two_level_split(int n, int& n1, int& n2) {
#define MC_TL_MATCH(A, B)      \
  if (n == (A) * (B)) {        \
    n1 = (A);                  \
    n2 = (B);                  \
    return true;               \
  }
  MC_TWO_LEVEL_LIST(MC_TL_MATCH)
#undef MC_TL_MATCH
  return false;
}

// Forward column launch with the radix-53 pairing the schedule asks for
template <int A, int B>
void launch_cols_fwd(const RowsFftArgs& a, bool paired, cudaStream_t st) {
  const dim3 grid(a.nrows, std::max(a.nfr, 1));
  const bool plain = a.n_out == A * B && a.keep_lo >= A * B && a.scale == 1.f;
  if constexpr (A == 53) {
    if (paired != kFwdColsPaired) {
      if (plain) k_rows_fft2l<A, B, false, !kFwdColsPaired, true><<<grid, TwoLevel<A, B>::T, 0, st>>>(a);
      else k_rows_fft2l<A, B, false, !kFwdColsPaired><<<grid, TwoLevel<A, B>::T, 0, st>>>(a);
      return;
    }
  }
  if (plain) k_rows_fft2l<A, B, false, kFwdColsPaired, true><<<grid, TwoLevel<A, B>::T, 0, st>>>(a);
  else k_rows_fft2l<A, B, false, kFwdColsPaired><<<grid, TwoLevel<A, B>::T, 0, st>>>(a);
}

cudaError_t launch_rows_fft2l(const RowsFftArgs& a, bool inverse, cudaStream_t st) {
  int n1 = 0, n2 = 0;
  if (!two_level_split(a.plan.n, n1, n2)) return cudaErrorInvalidValue;
  // the pairing of the radix-53 step (only N1 = 53 has one): schedule or built-in
  const bool paired = a.paired == 0 ? kFwdColsPaired : a.paired == 2;
#define MC_TL_LAUNCH(A, B)                                                                   \
  if (n1 == (A) && n2 == (B)) {                                                              \
    if (inverse)                                                                             \
      k_rows_fft2l<A, B, true, kFwdColsPaired><<<dim3(a.nrows, std::max(a.nfr, 1)), TwoLevel<A, B>::T, 0, st>>>(a); \
    else launch_cols_fwd<A, B>(a, paired, st);                                               \
    return cudaGetLastError();                                                               \
  }
  MC_TWO_LEVEL_LIST(MC_TL_LAUNCH)
#undef MC_TL_LAUNCH
  return cudaErrorInvalidValue;
}

}  // namespace mc
