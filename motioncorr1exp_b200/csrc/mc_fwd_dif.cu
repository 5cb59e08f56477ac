// Forward transforms of libmc for lengths 2N with a two-level N (sm_100a):
// 7420 = 2 x 3710 at -bin 2 (DFAlign.cu:710-806, cufunc.cu:162-176).
#include <algorithm>

#include "kcommon.cuh"

namespace mc {

// ---------------------------------------------------------------------------
// Lengths L = 2N with a two-level N (7420 = 2 x 3710 at -bin 2): one radix-2
// decimation-in-frequency step folded into the step-A loads,
//   A[m] = FFT_N(z_n + z_{n+N})[m] = Z[2m],
//   B[m] = FFT_N((z_n - z_{n+N}) W_L^n)[m] = Z[2m+1],
// then the two N-point two-level transforms, whose outputs go straight to
// the kept indices.  tw is the L-entry table exp(-2 pi i j / L), followed by
// the N-point transforms' own factors (fft_tables).

// Output pairs (k1, N1 - k1) of the N1-point step a radix-2 split transform
// needs when only its outputs below `lo` (2m < lo) and their mirror images
// (2m > L - lo) are kept: m = k2 + N2*k1 < lo/2 needs k1 <= (lo/2 - 1)/N2,
// one more pair for the boundary row; all pairs when that reaches (N1-1)/2.
template <int N1, int N2>
__device__ __forceinline__ int dif_kmax(int lo) {
  const int k = (lo / 2) / N2 + 1;
  return k < (N1 - 1) / 2 ? k : (N1 - 1) / 2;
}

// Forward rows of length L without references: two rows packed, read by the
// step-A loads.  Only the Z indices the half-spectrum split needs are kept,
// Z[0, hk) and Z(L - hk, L): the even ones, of the first transform, in a buffer
// of their own, the odd ones in the exchange buffer once the second transform
// has read it.  Without a Fourier crop the two ranges meet in Z[L / 2], which
// lies in the low one.  44.6 KB a CTA at 7420 -> 3710 (74 with the raw rows and every
// kept index staged): registers, not shared memory, set the four CTAs per SM.
// 24 frames of 7420^2 uint8 6.98 -> 6.69 ms (two output pairs of the pruned
// radix-53 step per loop pass: 6.66, with 72 bytes of spills; not taken).
template <int N1, int N2, typename Px>
__global__ void __launch_bounds__(TwoLevel<N1, N2>::T, 4) k_fwd_rows_dif(FwdRowsArgs a) {
  using TL = TwoLevel<N1, N2>;
  constexpr int N = TL::N, L = 2 * N;
  extern __shared__ float2 dyndif[];
  const int hk = a.hk, half = hk / 2 + 1;
  float2* zeven = dyndif;             // [2][half]: low, then high indices
  float2* ysm = dyndif + 2 * half;    // exchange buffer, later the odd indices
  float2* zodd = ysm;
  const int y0 = 2 * blockIdx.x, y1 = y0 + 1;
  float2* outA = a.outA + blockIdx.y * a.out_stride;
  const Px* f = reinterpret_cast<const Px*>(fwd_frame(a));
  const Px* p0 = f + (long long)(a.offy + y0) * a.nx + a.offx;
  const Px* p1 = f + (long long)(a.offy + y1) * a.nx + a.offx;
  const float2* tw = a.tw;
  auto keep = [&](float2* z, int idx, float2 v) {
    if (idx < hk) z[idx >> 1] = v;
    else if (idx > L - hk) z[half + ((idx - (L - hk + 1)) >> 1)] = v;
  };
  // wanted A/B outputs: m < hk/2 or m > N - hk/2, i.e. m = k2 + N2*k1 with
  // k1 or N1 - 1 - k1 at most (hk/2)/N2
  const int kmax = dif_kmax<N1, N2>(hk);
  TL::template run<false, false, false>(
      ysm, tw + L,
      [&](int n) {
        return make_float2((float)p0[n] + (float)p0[n + N], (float)p1[n] + (float)p1[n + N]);
      },
      [&](int m, float2 v) { keep(zeven, 2 * m, v); }, kmax);
  __syncthreads();
  TL::template run<false, true, false>(
      ysm, tw + L,
      [&](int n) {
        const float2 d = make_float2((float)p0[n] - (float)p0[n + N], (float)p1[n] - (float)p1[n + N]);
        return cmul(d, __ldg(tw + n));
      },
      [&](int m, float2 v) { keep(zodd, 2 * m + 1, v); }, kmax);
  __syncthreads();
  for (int k = threadIdx.x; k < hk; k += TL::T) {
    const float2* zs = k & 1 ? zodd : zeven;
    const float2 z = zs[k >> 1];
    const float2 zc = k == 0 || 2 * k == L ? z : zs[half + ((hk - 1 - k) >> 1)];  // Z[-k]
    const float2 X = make_float2(0.5f * (z.x + zc.x), 0.5f * (z.y - zc.y));
    const float2 Y = make_float2(0.5f * (z.y + zc.y), -0.5f * (z.x - zc.x));
    *reinterpret_cast<float4*>(outA + (long long)k * a.ldt + y0) = make_float4(X.x, X.y, Y.x, Y.y);
  }
}

// Forward columns of length L: out_row[i] = scale * X[i < keep_lo ? i : i + (L - n_out)].
// IN_PLACE (out = in, the columns of a movie that is not binned): the second
// transform reads the whole row again, so the first one's outputs wait in shared
// memory until the barrier inside the second has passed every read of the row.
// Uint8 movies, a frame's columns in place: 7420^2 288 us, 8192^2 243 (the
// mixed-radix engine, also safe in place: 535 and 376).
template <int N1, int N2, bool IN_PLACE>
__global__ void __launch_bounds__(TwoLevel<N1, N2>::T, 4) k_rows_fft_dif(RowsFftArgs a) {
  using TL = TwoLevel<N1, N2>;
  constexpr int N = TL::N, L = 2 * N;
  extern __shared__ float2 dyncol[];
  float2* ysm = dyncol;
  float2* zeven = dyncol + N;  // IN_PLACE: X[2m]
  const long long row = blockIdx.x;
  const float2* in = a.in + blockIdx.y * a.in_stride + row * a.ld_in;
  float2* out = a.out + blockIdx.y * a.out_stride + row * a.ld_out;
  const int shift = L - a.n_out, keep = a.keep_lo;
  const float sc = a.scale;
  const float2* tw = a.tw;
  auto get = [&](int i) { return IN_PLACE ? in[i] : __ldg(in + i); };
  auto put = [&](int i, float2 v) {
    int o;
    if (i < keep) o = i;
    else if (i >= keep + shift) o = i - shift;
    else return;
    out[o] = make_float2(v.x * sc, v.y * sc);
  };
  // wanted outputs i < keep or i >= keep + shift: with no crop all of them
  const int kmax = IN_PLACE || shift == 0 ? (N1 - 1) / 2 : dif_kmax<N1, N2>(keep + 1);
  TL::template run<false, false, false>(
      ysm, tw + L, [&](int n) { return cadd(get(n), get(n + N)); },
      [&](int m, float2 v) {
        if (IN_PLACE) zeven[m] = v;
        else put(2 * m, v);
      },
      kmax);
  __syncthreads();
  TL::template run<false, false, false>(
      ysm, tw + L,
      [&](int n) {
        const float2 x0 = get(n), x1 = get(n + N);
        return cmul(make_float2(x0.x - x1.x, x0.y - x1.y), __ldg(tw + n));
      },
      [&](int m, float2 v) { put(2 * m + 1, v); }, kmax);
  if (IN_PLACE)
    for (int m = threadIdx.x; m < N; m += TL::T) put(2 * m, zeven[m]);
}

bool dif_supported(int n) {
  int n1, n2;
  return n % 2 == 0 && two_level_split(n / 2, n1, n2);
}

cudaError_t launch_fwd_rows_dif(const FwdRowsArgs& a, cudaStream_t st) {
  int n1 = 0, n2 = 0;
  if (a.nu % 2 || !two_level_split(a.nu / 2, n1, n2)) return cudaErrorInvalidValue;
  const dim3 grid(a.nu / 2, std::max(a.nfr, 1));
#define MC_DIF_RAW(A, B, PX)                                                                          \
  {                                                                                                   \
    const size_t kept = 2 * (size_t)(a.hk / 2 + 1);                                                   \
    const size_t smem = (kept + std::max<size_t>((size_t)(A) * (B), kept)) * sizeof(float2);          \
    cudaError_t e = allow_smem((const void*)k_fwd_rows_dif<A, B, PX>, smem);                          \
    if (e != cudaSuccess) return e;                                                                   \
    k_fwd_rows_dif<A, B, PX><<<grid, TwoLevel<A, B>::T, smem, st>>>(a);                               \
    return cudaGetLastError();                                                                        \
  }
#define MC_DIF_LAUNCH(A, B)                                                                           \
  if (n1 == (A) && n2 == (B)) {                                                                       \
    switch (a.mode) {                                                                                 \
      case 0: MC_DIF_RAW(A, B, int8_t)                                                                \
      case MC_MODE_U8: MC_DIF_RAW(A, B, uint8_t)                                                      \
      case 1: MC_DIF_RAW(A, B, int16_t)                                                               \
      case 6: MC_DIF_RAW(A, B, uint16_t)                                                              \
      case MC_MODE_F16: MC_DIF_RAW(A, B, __half)                                                      \
      default: MC_DIF_RAW(A, B, float)                                                                \
    }                                                                                                 \
  }
  MC_TWO_LEVEL_LIST(MC_DIF_LAUNCH)
#undef MC_DIF_LAUNCH
#undef MC_DIF_RAW
  return cudaErrorInvalidValue;
}

template <int A, int B, bool IN_PLACE>
cudaError_t launch_cols_dif(const RowsFftArgs& a, cudaStream_t st) {
  const size_t smem = (IN_PLACE ? 2 : 1) * (size_t)A * B * sizeof(float2);
  cudaError_t e = allow_smem((const void*)k_rows_fft_dif<A, B, IN_PLACE>, smem);
  if (e != cudaSuccess) return e;
  k_rows_fft_dif<A, B, IN_PLACE><<<dim3(a.nrows, std::max(a.nfr, 1)), TwoLevel<A, B>::T, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_rows_fft_dif(const RowsFftArgs& a, cudaStream_t st) {
  int n1 = 0, n2 = 0;
  if (a.plan.n % 2 || !two_level_split(a.plan.n / 2, n1, n2)) return cudaErrorInvalidValue;
#define MC_DIF_LAUNCH(A, B) \
  if (n1 == (A) && n2 == (B)) return a.in == a.out ? launch_cols_dif<A, B, true>(a, st) : launch_cols_dif<A, B, false>(a, st);
  MC_TWO_LEVEL_LIST(MC_DIF_LAUNCH)
#undef MC_DIF_LAUNCH
  return cudaErrorInvalidValue;
}

}  // namespace mc
