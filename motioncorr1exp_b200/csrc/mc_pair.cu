// Pair stage of libmc (sm_100a): cross power x B-factor with the inverse
// along ky pruned to the pbx rows (cufunc.cu:343-370), and the pruned C2R
// along kx onto the pbx window (cufunc.cu:229-233, 404-407).
#include <algorithm>

// The column stage's Q-point codelets use packed FP32 FMAs in their odd-radix
// butterflies (bitwise the scalar results; 3 % faster here, while the
// forward kernels' 70-point codelets spill more with them).
#define MC_PACKED_FMA 1
#include "kcommon.cuh"

namespace mc {

// ============================================================ pair columns ==
// A CTA of 128 threads owns one column kx; it is split into teams of `team`
// threads (team = P rounded up to a warp multiple) and each team takes whole
// pairs.  Thread k1 < P of a team gathers its stride-P subsequence
// c(k1 + P*k2), k2 < Q, straight from the two spectra (coalesced over k1),
// runs the Q-point inverse FFT in registers, and parks the result in shared
// memory; the team then forms the pbx output rows as P-term sums.
constexpr int kRegThreads = 128;

__device__ __forceinline__ void team_barrier(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Resident 128-thread CTAs per SM the one-thread-per-subsequence kernel is
// compiled for: four (128 registers) up to Q = 40, three (168) up to 56, two
// (255) above.
constexpr int pair_reg_min_blocks(int Q) { return Q <= 40 ? 4 : (Q <= 56 ? 3 : 2); }

// ---- split n = P x Q fixed at compile time ----------------------------------
// The gather reads the stride-P subsequence at immediate offsets.  The outer
// sum out[m] = sum_k1 Y[r(m)][k1] W^(k1 y_m), r(m) = (ystart + m) mod Q, runs
// as items (output row m, chunk of at most 16 k1): Horner's rule from the
// chunk's last term down, acc = acc w + Y with w = W^(y_m) (4 FMAs per term,
// no twiddle loads; the powers of the rounded w drift by ~1e-6 over a chunk),
// then one multiply by W^(kb y_m).  A thread runs three items at a time with
// their chains interleaved (one item 5.85, two 5.71, three 5.64 ms per c2
// movie: with two warps per scheduler the dependent FMAs of one item left
// issue slots empty).  Consecutive threads take consecutive rows
// m, so their Y rows (odd stride in float2) fall on different bank pairs and
// their twiddle loads are contiguous.  The chunk partials meet in shared
// memory and are added in chunk order.
template <int Q, int P>
struct RpShape {
  static constexpr int T = P <= 32 ? 32 : (P <= 64 ? 64 : 128);  // team threads
  static constexpr int W = T / 32;                                // chunk count granule
  static constexpr int C = ((P + 15) / 16 + W - 1) / W * W;       // k1 chunks (96 C / T whole)
  static constexpr int L = (P + C - 1) / C;                       // chunk length <= 16
  static constexpr int PS = P | 1;                                // odd Y row stride (float2)
  static constexpr int YN = Q * PS;
};

size_t pair_cols_rp_smem(int n, int yn, int team, int chunks, int box) {
  const int teams = kRegThreads / team;
  return (size_t)((n + 1) / 2) * sizeof(float2) + (size_t)(chunks + 1) * box * sizeof(float2) +
         (size_t)teams * ((size_t)yn + (size_t)chunks * box) * sizeof(float2);
}

template <int Q, int P>
__global__ void __launch_bounds__(kRegThreads, pair_reg_min_blocks(Q)) k_pair_cols_rp(PairColsArgs a) {
  using S = RpShape<Q, P>;
  constexpr int T = S::T, C = S::C, L = S::L, N = P * Q, PS = S::PS, YN = S::YN;
  extern __shared__ float2 sm[];
  const int box = a.box;
  float* wcol = reinterpret_cast<float*>(sm);
  // twiddle rows the sums need: tws[0][m] = W^(y_m) (twO row 1), tws[1 + c][m]
  // = W^(kb(c) y_m) (twO row c L)
  float2* tws = sm + (N + 1) / 2;
  constexpr int teams = kRegThreads / T;
  const int tid = threadIdx.x;
  const int tm = tid / T, lt = tid - tm * T;
  float2* Y = tws + (C + 1) * box + (size_t)tm * (YN + C * box);
  float2* part = Y + YN;
  const int kx = blockIdx.y;
  for (int ky = tid; ky < N; ky += kRegThreads) {
    const int y = ky < N / 2 ? ky : ky - N;
    wcol[ky] = expf(a.mbf * (float)(kx * kx + y * y)) * a.inv_size;
  }
  for (int i = tid; i < (C + 1) * box; i += kRegThreads) {
    const int row = i / box, m = i - row * box;
    const int k = row == 0 ? 1 : min((row - 1) * L, P - 1);
    tws[i] = __ldg(a.twO + (long long)k * box + m);
  }
  __syncthreads();
  const int ys = a.ystart % Q;
  const int p0 = blockIdx.x * a.pairs_per_cta;
  const int p1 = min(p0 + a.pairs_per_cta, a.npairs);
  for (int p = p0 + tm; p < p1; p += teams) {
    const int2 pr = a.pairs[p];
    if (lt < P) {
      const float2* ca = a.specA + (long long)pr.x * a.strideA + (long long)kx * a.ldn + lt;
      const float2* cb = a.specB + (long long)pr.y * a.strideB + (long long)kx * a.ldn + lt;
      const float* wc = wcol + lt;
      float2 x[Q];
#pragma unroll
      for (int k2 = 0; k2 < Q; k2++) x[k2] = cscale(cmulc(__ldg(ca + P * k2), __ldg(cb + P * k2)), wc[P * k2]);
      fft_reg_pf<Q, true>(x);
#pragma unroll
      for (int r = 0; r < Q; r++) Y[lt + PS * r] = x[r];
    }
    team_barrier(1 + tm, T);
    int c = lt / box, m = lt - (lt / box) * box;
    // three items per pass, their chains interleaved (three times the
    // independent work)
    for (int it = lt; it < box * C; it += 3 * T) {
      int c1 = c, m1 = m + T;
      while (m1 >= box) {
        m1 -= box;
        c1++;
      }
      int c2 = c1, m2 = m1 + T;
      while (m2 >= box) {
        m2 -= box;
        c2++;
      }
      const bool has1 = it + T < box * C, has2 = it + 2 * T < box * C;
      const int nc_ = c2, nm_ = m2;
      if (!has1) {
        c1 = c;
        m1 = m;
      }
      if (!has2) {
        c2 = c;
        m2 = m;
      }
      int r0 = ys + m % Q, r1 = ys + m1 % Q, r2 = ys + m2 % Q;
      if (r0 >= Q) r0 -= Q;
      if (r1 >= Q) r1 -= Q;
      if (r2 >= Q) r2 -= Q;
      const int kb0 = c * L, kb1 = c1 * L, kb2 = c2 * L;
      const float2* yr0 = Y + PS * r0 + kb0;
      const float2* yr1 = Y + PS * r1 + kb1;
      const float2* yr2 = Y + PS * r2 + kb2;
      const float2 w0 = tws[m], w1 = tws[m1], w2 = tws[m2];
      const float2 v0 = cmul(w0, w0), v1 = cmul(w1, w1), v2 = cmul(w2, w2);
      float2 ae0 = make_float2(0.f, 0.f), ao0 = make_float2(0.f, 0.f);
      float2 ae1 = make_float2(0.f, 0.f), ao1 = make_float2(0.f, 0.f);
      float2 ae2 = make_float2(0.f, 0.f), ao2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int kk = L - 1; kk >= 0; kk--) {
        if (L * C == P || kb0 + kk < P) {
          const float2 yv = yr0[kk];
          float2& h = (kk & 1) ? ao0 : ae0;
          const float2 s = h;
          h.x = fmaf(s.x, v0.x, fmaf(-s.y, v0.y, yv.x));
          h.y = fmaf(s.x, v0.y, fmaf(s.y, v0.x, yv.y));
        }
        if (L * C == P || kb1 + kk < P) {
          const float2 yv = yr1[kk];
          float2& h = (kk & 1) ? ao1 : ae1;
          const float2 s = h;
          h.x = fmaf(s.x, v1.x, fmaf(-s.y, v1.y, yv.x));
          h.y = fmaf(s.x, v1.y, fmaf(s.y, v1.x, yv.y));
        }
        if (L * C == P || kb2 + kk < P) {
          const float2 yv = yr2[kk];
          float2& h = (kk & 1) ? ao2 : ae2;
          const float2 s = h;
          h.x = fmaf(s.x, v2.x, fmaf(-s.y, v2.y, yv.x));
          h.y = fmaf(s.x, v2.y, fmaf(s.y, v2.x, yv.y));
        }
      }
      float2 acc0, acc1, acc2;
      acc0.x = fmaf(ao0.x, w0.x, fmaf(-ao0.y, w0.y, ae0.x));
      acc0.y = fmaf(ao0.x, w0.y, fmaf(ao0.y, w0.x, ae0.y));
      acc1.x = fmaf(ao1.x, w1.x, fmaf(-ao1.y, w1.y, ae1.x));
      acc1.y = fmaf(ao1.x, w1.y, fmaf(ao1.y, w1.x, ae1.y));
      acc2.x = fmaf(ao2.x, w2.x, fmaf(-ao2.y, w2.y, ae2.x));
      acc2.y = fmaf(ao2.x, w2.y, fmaf(ao2.y, w2.x, ae2.y));
      if (kb0 < P) acc0 = cmul(acc0, tws[(1 + c) * box + m]);
      if (kb1 < P) acc1 = cmul(acc1, tws[(1 + c1) * box + m1]);
      if (kb2 < P) acc2 = cmul(acc2, tws[(1 + c2) * box + m2]);
      part[c * box + m] = acc0;
      if (has1) part[c1 * box + m1] = acc1;
      if (has2) part[c2 * box + m2] = acc2;
      m = nm_ + T;
      c = nc_;
      while (m >= box) {
        m -= box;
        c++;
      }
    }
    team_barrier(1 + tm, T);
    for (int m = lt; m < box; m += T) {
      float2 s = part[m];
#pragma unroll
      for (int c = 1; c < C; c++) s = cadd(s, part[c * box + m]);
      a.G[((long long)p * a.H + kx) * box + m] = s;
    }
    // the next pair writes Y before its first barrier and part after it:
    // every read of this pair's Y precedes the second barrier above, and every
    // read of part precedes the next pair's first barrier
  }
}

// ---- row stage with the same compiled split --------------------------------
// box[p][yb][xb] = sum_kx h(kx) Re(G[p][kx][yb] exp(+2 pi i kx x_xb / n)) is
// the length-n inverse DFT of the Hermitian extension of row yb (real parts
// at kx = 0 and n/2, conj(G[n - kx]) above n/2), evaluated at the box's
// columns.  Two rows ride in one complex sequence z = Ga + i Gb, so the real
// and imaginary parts of the result are the two output rows.  A CTA stages
// G[p][:, 2 teams rows] (coalesced, odd row stride), each team gathers its
// row pair, runs the inverse Q-point codelet on the stride-P subsequences and
// forms the box columns by the column stage's Horner sums.
template <int Q, int P>
__host__ __device__ __forceinline__ size_t pair_rows_rp_region(int H) {
  using S = RpShape<Q, P>;
  constexpr int teams = kRegThreads / S::T;
  const size_t g = (size_t)H * (2 * teams + 1);
  const size_t y = (size_t)teams * S::YN;
  return g > y ? g : y;
}

template <int Q, int P>
size_t pair_rows_rp_smem(int H, int box) {
  using S = RpShape<Q, P>;
  constexpr int teams = kRegThreads / S::T;
  return (pair_rows_rp_region<Q, P>(H) + (size_t)(S::C + 1) * box + (size_t)teams * S::C * box) * sizeof(float2);
}

template <int Q, int P>
__global__ void __launch_bounds__(kRegThreads, pair_reg_min_blocks(Q)) k_pair_rows_rp(PairRowsArgs a, const float2* __restrict__ twO,
                                                                                        int ystart) {
  using S = RpShape<Q, P>;
  constexpr int T = S::T, C = S::C, L = S::L, N = P * Q, PS = S::PS;
  constexpr int teams = kRegThreads / T, R = 2 * teams, RS = R + 1;
  extern __shared__ float2 sm[];
  const int box = a.box, H = a.H;
  float2* reg = sm;                                    // staged G rows, then the teams' Y
  float2* tws = sm + pair_rows_rp_region<Q, P>(H);
  float2* part0 = tws + (C + 1) * box;
  const int tid = threadIdx.x, tm = tid / T, lt = tid - tm * T;
  const int p = blockIdx.x, yb0 = blockIdx.y * R;
  const float2* G = a.G + (long long)p * H * box;
  if (!(box & 1) && yb0 + R <= box) {
    // two rows a 16-byte load, eight in flight a thread: the staging, not the
    // transforms, set the pace one element at a time (378 pairs of
    // 3710^2 491 -> 397 us, 129 of 4096^2 154 -> 122, 55 of 1024^2 23 -> 19)
#pragma unroll 8
    for (int i = tid; i < H * (R / 2); i += kRegThreads) {
      const int kx = i / (R / 2), r = 2 * (i - kx * (R / 2));
      const float4 v = __ldg(reinterpret_cast<const float4*>(G + kx * box + yb0 + r));
      reg[kx * RS + r] = make_float2(v.x, v.y);
      reg[kx * RS + r + 1] = make_float2(v.z, v.w);
    }
  } else {
    for (int i = tid; i < H * R; i += kRegThreads) {
      const int kx = i / R, r = i - kx * R;
      reg[kx * RS + r] = yb0 + r < box ? G[(long long)kx * box + yb0 + r] : make_float2(0.f, 0.f);
    }
  }
  for (int i = tid; i < (C + 1) * box; i += kRegThreads) {
    const int row = i / box, m = i - row * box;
    const int k = row == 0 ? 1 : min((row - 1) * L, P - 1);
    tws[i] = __ldg(twO + (long long)k * box + m);
  }
  __syncthreads();
  float2 x[Q];
  if (lt < P) {
    const int ra = 2 * tm, rb = ra + 1;
#pragma unroll
    for (int k2 = 0; k2 < Q; k2++) {
      const int kx = lt + P * k2;
      float2 z;
      if (kx == 0 || 2 * kx == N) {
        z = make_float2(reg[kx * RS + ra].x, reg[kx * RS + rb].x);
      } else if (2 * kx < N) {
        const float2 ga = reg[kx * RS + ra], gb = reg[kx * RS + rb];
        z = make_float2(ga.x - gb.y, ga.y + gb.x);
      } else {
        const int kr = N - kx;
        const float2 ga = reg[kr * RS + ra], gb = reg[kr * RS + rb];
        z = make_float2(ga.x + gb.y, gb.x - ga.y);
      }
      x[k2] = z;
    }
    fft_reg_pf<Q, true>(x);
  }
  __syncthreads();  // every team has gathered: the staged rows give way to Y
  float2* Y = reg + (size_t)tm * S::YN;
  float2* part = part0 + (size_t)tm * C * box;
  if (lt < P) {
#pragma unroll
    for (int r = 0; r < Q; r++) Y[lt + PS * r] = x[r];
  }
  team_barrier(1 + tm, T);
  const int ys = ystart % Q;
  int c = lt / box, m = lt - (lt / box) * box;
  for (int it = lt; it < box * C; it += T) {
    int r = ys + m % Q;
    if (r >= Q) r -= Q;
    const int kb = c * L;
    const float2* yr = Y + PS * r + kb;
    const float2 w = tws[m];
    const float2 w2 = cmul(w, w);
    float2 ae = make_float2(0.f, 0.f), ao = make_float2(0.f, 0.f);
#pragma unroll
    for (int kk = L - 1; kk >= 0; kk--) {
      if (L * C == P || kb + kk < P) {
        const float2 yv = yr[kk];
        float2& h = (kk & 1) ? ao : ae;
        const float2 s = h;
        h.x = fmaf(s.x, w2.x, fmaf(-s.y, w2.y, yv.x));
        h.y = fmaf(s.x, w2.y, fmaf(s.y, w2.x, yv.y));
      }
    }
    float2 acc;
    acc.x = fmaf(ao.x, w.x, fmaf(-ao.y, w.y, ae.x));
    acc.y = fmaf(ao.x, w.y, fmaf(ao.y, w.x, ae.y));
    if (kb < P) acc = cmul(acc, tws[(1 + c) * box + m]);
    else acc = make_float2(0.f, 0.f);
    part[c * box + m] = acc;
    m += T;
    while (m >= box) {
      m -= box;
      c++;
    }
  }
  team_barrier(1 + tm, T);
  const int ya = yb0 + 2 * tm, yb = ya + 1;
  const int o = a.order ? a.order[p] : p;
  for (int mm = lt; mm < box; mm += T) {
    float2 s = part[mm];
#pragma unroll
    for (int cc = 1; cc < C; cc++) s = cadd(s, part[cc * box + mm]);
    if (ya < box) a.boxes[((long long)o * box + ya) * box + mm] = s.x;
    if (yb < box) a.boxes[((long long)o * box + yb) * box + mm] = s.y;
  }
}

// the compiled (Q, P) splits of the tuned lengths: 3710, 4096, 2048, 1024
#define MC_RP_LIST(X) X(35, 106) X(70, 53) X(64, 64) X(32, 128) X(64, 32) X(32, 64) X(16, 128) X(32, 32) X(16, 64)

size_t pair_cols_launch_smem(int n, int P, int Q, int box) {
#define MC_RP_SMEM(A, B) \
  if (Q == (A) && P == (B)) return pair_cols_rp_smem(n, RpShape<A, B>::YN, RpShape<A, B>::T, RpShape<A, B>::C, box);
  MC_RP_LIST(MC_RP_SMEM)
#undef MC_RP_SMEM
  return pair_cols_smem(n, P, Q, box);
}

bool pair_cols_reg_supported(int P, int Q) {
  if (P < 1 || P > kRegThreads) return false;
  for (int q : kCodelets)
    if (q == Q) return true;
  return false;
}

cudaError_t launch_pair_cols_pruned(const PairColsArgs& c, cudaStream_t st);

cudaError_t launch_pair_cols(const PairColsArgs& a, cudaStream_t st) {
  const int ppc = a.pairs_per_cta > 0 ? a.pairs_per_cta : 32;
  dim3 grid((a.npairs + ppc - 1) / ppc, a.H);
#define MC_RP_LAUNCH(A, B)                                                                                  \
  if (a.Q == (A) && a.P == (B) && a.n == (A) * (B)) {                                                      \
    const size_t smem = pair_cols_rp_smem(a.n, RpShape<A, B>::YN, RpShape<A, B>::T, RpShape<A, B>::C, a.box); \
    cudaError_t e = allow_smem((const void*)k_pair_cols_rp<A, B>, smem);                                   \
    if (e != cudaSuccess) return e;                                                                        \
    PairColsArgs b = a;                                                                                    \
    b.pairs_per_cta = ppc;                                                                                 \
    k_pair_cols_rp<A, B><<<grid, kRegThreads, smem, st>>>(b);                                              \
    return cudaGetLastError();                                                                             \
  }
  MC_RP_LIST(MC_RP_LAUNCH)
#undef MC_RP_LAUNCH
  return launch_pair_cols_pruned(a, st);
}

// =============================================================== pair rows ==
// Sizes without a compiled split: the product box[yb][xb] = sum_kx G.x cs.x -
// G.y cs.y, kx ascending.  A CTA of 64 threads forms an 8 RI x 32 tile of one
// pair's window, RI x 4 outputs a thread from 16-byte shared-memory reads;
// chunks of kRowK kx are staged through shared memory, the next chunk's loads
// in flight while the current one is summed.  FP32 issue bounds it when the
// tiles of all pairs fill the GPU, latency when they do not (launch_pair_rows).
// Measured against one CTA per pair with 6 x 6 outputs a thread: 21 pairs of
// 256^2 37 -> 13 us, 153 pairs of 520^2 100 -> 42, 105 pairs of 1500^2 254 ->
// 142, 55 pairs of 4092^2 681 -> 228.
constexpr int kRowTile = 32;
constexpr int kRowK = 16;
constexpr int kRowThreads = 64;

template <int RI>
__global__ void __launch_bounds__(kRowThreads) k_pair_rows(PairRowsArgs a) {
  constexpr int TY = 8 * RI;                         // tile rows
  constexpr int EC = kRowK * kRowTile / kRowThreads;  // elements a thread stages of cs
  constexpr int EG = kRowK * TY / kRowThreads;        // and of G
  __shared__ __align__(16) float2 gs[2][kRowK][TY];
  __shared__ __align__(16) float2 cs[2][kRowK][kRowTile];
  const int box = a.box, tid = threadIdx.x;
  const int tiles = (box + kRowTile - 1) / kRowTile;
  const int yb0 = (blockIdx.x / tiles) * TY, xb0 = (blockIdx.x % tiles) * kRowTile, p = blockIdx.y;
  // rows ty .. ty + RI - 1; columns tx, tx + 1, tx + 16, tx + 17 (16-byte reads of
  // eight neighbouring threads fall on distinct banks)
  const int ty = (tid >> 3) * RI, tx = (tid & 7) * 2;
  const float2* G = a.G + (long long)p * a.H * box;
  const int cc = tid % kRowTile, ck = tid / kRowTile, gc = tid % TY, gk = tid / TY;
  const bool gok = yb0 + gc < box, cok = xb0 + cc < box;
  float2 gr[EG], cr[EC];
  auto fetch = [&](int kx0) {
#pragma unroll
    for (int i = 0; i < EG; i++) {
      const int kx = kx0 + gk + i * (kRowThreads / TY);
      gr[i] = kx < a.H && gok ? __ldg(G + (long long)kx * box + yb0 + gc) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < EC; i++) {
      const int kx = kx0 + ck + i * (kRowThreads / kRowTile);
      cr[i] = kx < a.H && cok ? __ldg(a.cs + (long long)kx * box + xb0 + cc) : make_float2(0.f, 0.f);
    }
  };
  auto park = [&](int s) {
#pragma unroll
    for (int i = 0; i < EG; i++) gs[s][gk + i * (kRowThreads / TY)][gc] = gr[i];
#pragma unroll
    for (int i = 0; i < EC; i++) cs[s][ck + i * (kRowThreads / kRowTile)][cc] = cr[i];
  };
  float acc[RI][4];
#pragma unroll
  for (int i = 0; i < RI; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  fetch(0);
  park(0);
  __syncthreads();
  for (int kx0 = 0, s = 0; kx0 < a.H; kx0 += kRowK, s ^= 1) {
    const bool more = kx0 + kRowK < a.H;
    if (more) fetch(kx0 + kRowK);
#pragma unroll
    for (int kk = 0; kk < kRowK; kk++) {
      float2 g[RI];
#pragma unroll
      for (int i = 0; i < RI; i += 2) {
        const float4 v = *reinterpret_cast<const float4*>(&gs[s][kk][ty + i]);
        g[i] = make_float2(v.x, v.y);
        g[i + 1] = make_float2(v.z, v.w);
      }
      const float4 c0 = *reinterpret_cast<const float4*>(&cs[s][kk][tx]);
      const float4 c1 = *reinterpret_cast<const float4*>(&cs[s][kk][tx + 16]);
      const float2 w[4] = {{c0.x, c0.y}, {c0.z, c0.w}, {c1.x, c1.y}, {c1.z, c1.w}};
#pragma unroll
      for (int i = 0; i < RI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(g[i].x, w[j].x, fmaf(-g[i].y, w[j].y, acc[i][j]));
    }
    if (more) park(s ^ 1);
    __syncthreads();
  }
  const long long o = a.order ? a.order[p] : p;
#pragma unroll
  for (int i = 0; i < RI; i++) {
    const int yb = yb0 + ty + i;
    if (yb >= box) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int xb = xb0 + tx + (j & 1) + (j >> 1) * 16;
      if (xb < box) a.boxes[(o * box + yb) * box + xb] = acc[i][j];
    }
  }
}

cudaError_t launch_pair_rows(const PairRowsArgs& a, cudaStream_t st) {
  if (a.twO) {
#define MC_RP_ROWS(A, B)                                                                            \
  if (a.Q == (A) && a.P == (B) && 2 * (a.H - 1) == (A) * (B)) {                                    \
    constexpr int rows = 2 * (kRegThreads / RpShape<A, B>::T);                                     \
    const size_t smem = pair_rows_rp_smem<A, B>(a.H, a.box);                                       \
    if (smem > 227 * 1024) return cudaErrorInvalidValue;                                            \
    cudaError_t e = allow_smem((const void*)k_pair_rows_rp<A, B>, smem);                           \
    if (e != cudaSuccess) return e;                                                                 \
    k_pair_rows_rp<A, B><<<dim3(a.npairs, (a.box + rows - 1) / rows), kRegThreads, smem, st>>>(a, a.twO, a.ystart); \
    return cudaGetLastError();                                                                      \
  }
    MC_RP_LIST(MC_RP_ROWS)
#undef MC_RP_ROWS
  }
  // two rows a thread instead of four while the larger tiles would leave an SM
  // fewer than four CTAs (two warps each): 21 pairs of 256^2, box 64, 13.3 us
  // against 16.1; 55 pairs of 4092^2 226 / 228; 105 pairs of 1500^2 154 / 142
  const int tiles = (a.box + kRowTile - 1) / kRowTile;
  if (tiles * tiles * a.npairs < 148 * 4)
    k_pair_rows<2><<<dim3(tiles * ((a.box + 15) / 16), a.npairs), kRowThreads, 0, st>>>(a);
  else
    k_pair_rows<4><<<dim3(tiles * tiles, a.npairs), kRowThreads, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace mc
