// Column stage of the pair kernels for splits n = P*Q that are not compiled in
// (mc_pair.cu holds those): cross power x B-factor, inverse along ky kept on
// the box rows (cufunc.cu:343-370).
//
// A unit is one (pair, kx) column c(ky).  Its P stride-P subsequences
// c(k1 + P k2) go through Q-point inverse FFTs, and
//     out[m] = sum_k1 Y[r(m)][k1] W^(k1 y_m),  y_m = (ystart + m) mod n,
//     r(m) = (ystart + m) mod Q,  W = exp(2 pi i / n)
// runs as two sums (k1 below and from (P + 1) / 2) with exact factors.  What
// bounds the sums is their shared-memory and table reads, two for four FMAs,
// so a thread forms one (m, half) of several units at once: one factor serves
// kSumUnits of them.
//
// Q a codelet length: one thread per subsequence holds its Q values in
// registers, and a CTA takes as many units at once as fill its 128 threads (P
// = 4 used 4 of 32 threads before).  Other Q (template 0): the mixed-radix
// engine over shared memory, 256 threads.
// Measured, one unit per warp team (or per 256 threads for the engine) before
// and now: 21 pairs of 256^2 42 -> 16 us, 153 pairs of 520^2 130 -> 72, 105
// pairs of 1500^2 625 -> 377, 55 pairs of 4092^2 (engine) 5.12 -> 2.47 ms.
#include <algorithm>

#define MC_PACKED_FMA 1
#include "kcommon.cuh"

namespace mc {

struct PrunedArgs {
  int n, H, box, P, Q, ystart;
  int PS;           // odd pitch of a Y row
  int NU;           // units a CTA holds at once
  int per_cta;      // units a CTA takes in turn
  int table;        // 1: the factors W^(k1 y_m) are staged in shared memory
  FastDiv pdiv, boxdiv, qdiv;
  const float2* twO;  // [P][box] W^(k1 y_m)
  FftPlan1D qplan;    // Q = 0 template
  const float2* twQ;
  const float2 *specA, *specB;
  long long strideA, strideB;
  const int2* pairs;
  int npairs, ldn;
  float mbf, inv_size;
  float2* G;        // [npairs][H][box]
};

constexpr int kSumUnits = 4;
constexpr int pruned_threads(int Q) { return Q ? 128 : 384; }  // the most a CTA has
// Resident CTAs a codelet kernel is compiled for: four (128 registers) up to
// Q = 40, three (168) up to 56, two (255) above.
constexpr int pruned_min_blocks(int Q) { return Q == 0 ? 2 : (Q <= 40 ? 4 : (Q <= 56 ? 3 : 2)); }

// U units' sums of one (m, half): y at the half's first term of the first unit
template <int U, bool STAGED>
__device__ __forceinline__ void half_sums(const float2* y, int unit, const float2* tw, int box, int cnt, float2* acc) {
#pragma unroll
  for (int u = 0; u < U; u++) acc[u] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < cnt; k++) {
    const float2 t = STAGED ? tw[k * box] : __ldg(tw + (long long)k * box);
#pragma unroll
    for (int u = 0; u < U; u++) {
      const float2 v = y[u * unit + k];
      acc[u].x = fmaf(t.x, v.x, fmaf(-t.y, v.y, acc[u].x));
      acc[u].y = fmaf(t.x, v.y, fmaf(t.y, v.x, acc[u].y));
    }
  }
}

template <bool STAGED>
__device__ __forceinline__ void unit_sums(int left, const float2* y, int unit, const float2* tw, int box, int cnt,
                                          float2* acc) {
  if (left >= 4) half_sums<4, STAGED>(y, unit, tw, box, cnt, acc);
  else if (left == 3) half_sums<3, STAGED>(y, unit, tw, box, cnt, acc);
  else if (left == 2) half_sums<2, STAGED>(y, unit, tw, box, cnt, acc);
  else half_sums<1, STAGED>(y, unit, tw, box, cnt, acc);
}

template <int QT>
__global__ void __launch_bounds__(pruned_threads(QT), pruned_min_blocks(QT)) k_pair_cols_pruned(PrunedArgs a) {
  const int NT = QT ? pruned_threads(QT) : (int)blockDim.x;
  extern __shared__ float2 sm[];
  const int n = a.n, P = a.P, box = a.box, PS = a.PS;
  const int Q = QT ? QT : a.Q;
  const int tid = threadIdx.x;
  const int unit = Q * PS;  // float2 of one unit's Y
  float2* Y0 = sm;
  float2* Y1 = QT || Q == 1 ? sm : sm + (size_t)a.NU * unit;  // the engine's second buffer
  float2* part = Y1 + (size_t)a.NU * unit;           // [NU][2][box]
  // the units' two columns, read by every load of the engine's first pass
  float2* tws = part + (size_t)a.NU * 2 * box;        // [P][box] (a.table)
  const float2** cols = reinterpret_cast<const float2**>(tws + (a.table ? P * box : 0));
  int* rofs = reinterpret_cast<int*>(cols + 2 * a.NU);
  float* wcol = reinterpret_cast<float*>(rofs + box);  // B-factor weights of this kx
  const int kx = blockIdx.y;
  for (int m = tid; m < box; m += NT) {
    uint32_t q, r;
    fdivmod((uint32_t)(a.ystart + m), a.qdiv, q, r);
    rofs[m] = (int)r * PS;
  }
  if (a.table)
    for (int i = tid; i < P * box; i += NT) tws[i] = __ldg(a.twO + i);
  for (int ky = tid; ky < n; ky += NT) {
    const int y = ky < n / 2 ? ky : ky - n;
    wcol[ky] = expf(a.mbf * (float)(kx * kx + y * y)) * a.inv_size;
  }
  __syncthreads();
  const int u0 = blockIdx.x * a.per_cta, u1 = min(u0 + a.per_cta, a.npairs);
  auto column = [&](int u, const float2*& ca, const float2*& cb) {
    const int2 pr = a.pairs[u];
    ca = a.specA + (long long)pr.x * a.strideA + (long long)kx * a.ldn;
    cb = a.specB + (long long)pr.y * a.strideB + (long long)kx * a.ldn;
  };
  auto product = [&](const float2* ca, const float2* cb, int ky) {
    return cscale(cmulc(__ldg(ca + ky), __ldg(cb + ky)), wcol[ky]);
  };
  uint32_t tq = 0, tk = 0;  // this thread's (unit, subsequence)
  if constexpr (QT > 0) fdivmod((uint32_t)tid, a.pdiv, tq, tk);
  const int khalf = (P + 1) / 2;
  for (int g = u0; g < u1; g += a.NU) {
    const int nu = min(a.NU, u1 - g);
    const float2* Y = Y0;
    if constexpr (QT == 0) {
      if (tid < nu) column(g + tid, cols[2 * tid], cols[2 * tid + 1]);
      __syncthreads();
    }
    if constexpr (QT > 0) {
      if ((int)tq < nu) {
        const float2 *ca, *cb;
        column(g + (int)tq, ca, cb);
        float2 x[QT ? QT : 1];
#pragma unroll
        for (int k2 = 0; k2 < QT; k2++) x[k2] = product(ca, cb, (int)tk + P * k2);
        fft_reg_pf<QT, true>(x);
        float2* y = Y0 + tq * unit + tk;
#pragma unroll
        for (int r = 0; r < QT; r++) y[r * PS] = x[r];
      }
    } else if (Q == 1) {
      for (int q = 0; q < nu; q++) {
        const float2 *ca = cols[2 * q], *cb = cols[2 * q + 1];
        for (int ky = tid; ky < n; ky += NT) Y0[q * unit + ky] = product(ca, cb, ky);
      }
    } else {
      fft_exec<true, true>(
          Y0, Y1, a.qplan, a.NU * P, 0, a.twQ, tid, NT,
          [&](int b, int i) {
            uint32_t q = 0, k1 = (uint32_t)b;
            if (a.NU > 1) fdivmod((uint32_t)b, a.pdiv, q, k1);
            if ((int)q >= nu) return make_float2(0.f, 0.f);
            return product(cols[2 * q], cols[2 * q + 1], (int)k1 + P * i);
          },
          [&](float2* dst, int b, int i, float2 v) {
            uint32_t q = 0, k1 = (uint32_t)b;
            if (a.NU > 1) fdivmod((uint32_t)b, a.pdiv, q, k1);
            dst[q * unit + i * PS + k1] = v;
          });
      if (!(a.qplan.nst & 1)) Y = Y1;
    }
    __syncthreads();
    // items (group of units, half, output row), row fastest
    const int groups = (nu + kSumUnits - 1) / kSumUnits, total = groups * 2 * box;
    for (int it = tid; it < total; it += NT) {
      uint32_t gh, m;
      fdivmod((uint32_t)it, a.boxdiv, gh, m);
      const int h = (int)gh & 1, q0 = (int)(gh >> 1) * kSumUnits, left = nu - q0;
      const int k0 = h ? khalf : 0, cnt = h ? P - khalf : khalf;
      const float2* y = Y + q0 * unit + rofs[m] + k0;
      float2 acc[kSumUnits];
      if (a.table) unit_sums<true>(left, y, unit, tws + k0 * box + m, box, cnt, acc);
      else unit_sums<false>(left, y, unit, a.twO + (long long)k0 * box + m, box, cnt, acc);
#pragma unroll
      for (int u = 0; u < kSumUnits; u++)
        if (u < left) part[((q0 + u) * 2 + h) * box + m] = acc[u];
    }
    __syncthreads();
    for (int i = tid; i < nu * box; i += NT) {
      uint32_t q, m;
      fdivmod((uint32_t)i, a.boxdiv, q, m);
      const float2* s = part + q * 2 * box + m;
      a.G[((long long)(g + (int)q) * a.H + kx) * box + m] = cadd(s[0], s[box]);
    }
    // the next units' partials are written behind their first barrier
  }
}

template <int QT>
cudaError_t launch_pruned_q(const PrunedArgs& a, size_t smem, dim3 grid, int threads, cudaStream_t st) {
  cudaError_t e = allow_smem((const void*)k_pair_cols_pruned<QT>, smem);
  if (e != cudaSuccess) return e;
  k_pair_cols_pruned<QT><<<grid, threads, smem, st>>>(a);
  return cudaGetLastError();
}

template <int I = 0>
cudaError_t dispatch_pruned(const PrunedArgs& a, int Q, size_t smem, dim3 grid, int threads, cudaStream_t st) {
  if constexpr (I < kNumCodelets) {
    constexpr int C = kCodelets[I];
    if (Q == C) return launch_pruned_q<C>(a, smem, grid, threads, st);
    return dispatch_pruned<I + 1>(a, Q, smem, grid, threads, st);
  } else {
    return launch_pruned_q<0>(a, smem, grid, threads, st);
  }
}


namespace {

// the codelet length the kernel template takes, or 0
int pruned_template(int P, int Q) { return pair_cols_reg_supported(P, Q) ? Q : 0; }

size_t pruned_smem(int n, int P, int Q, int box, int NU) {
  const int buffers = pruned_template(P, Q) || Q == 1 ? 1 : 2;
  return sizeof(float2) * (size_t)NU * ((size_t)buffers * Q * (P | 1) + 2 * (size_t)box) +
         2 * sizeof(void*) * (size_t)NU + sizeof(int) * (size_t)box + sizeof(float) * (size_t)n;
}

}  // namespace

size_t pair_cols_smem(int n, int P, int Q, int box) { return pruned_smem(n, P, Q, box, 1); }

cudaError_t launch_pair_cols_pruned(const PairColsArgs& c, cudaStream_t st) {
  const int qt = pruned_template(c.P, c.Q);
  PrunedArgs a{};
  a.n = c.n;
  a.H = c.H;
  a.box = c.box;
  a.P = c.P;
  a.Q = c.Q;
  a.ystart = c.ystart;
  a.twO = c.twO;
  a.qplan = c.qplan;
  a.twQ = c.twQ;
  a.specA = c.specA;
  a.specB = c.specB;
  a.strideA = c.strideA;
  a.strideB = c.strideB;
  a.pairs = c.pairs;
  a.npairs = c.npairs;
  a.ldn = c.ldn;
  a.mbf = c.mbf;
  a.inv_size = c.inv_size;
  a.G = c.G;
  a.PS = c.P | 1;
  // units side by side: as many as fill the threads (codelets) or give the
  // engine's stages 4096 elements, within the shared memory of the CTAs the
  // kernel is compiled for
  const int want = std::max(1, qt ? pruned_threads(qt) / a.P : 4096 / a.n);
  const size_t cap = 227 * 1024 / pruned_min_blocks(qt) - 1024;
  a.NU = std::min(want, a.npairs);
  while (a.NU > 1 && pruned_smem(a.n, a.P, a.Q, a.box, a.NU) > cap) a.NU--;
  size_t smem = pruned_smem(a.n, a.P, a.Q, a.box, a.NU);
  const size_t tab = sizeof(float2) * (size_t)a.P * a.box;
  // the sums' factors in shared memory where that costs no resident CTA (105
  // pairs of 1500^2: 413 us reading them through L1, 376 staged)
  a.table = smem + tab <= cap;
  if (a.table) smem += tab;
  int threads = pruned_threads(qt);
  if (!qt && a.Q > 1) {
    // the engine's passes have n / R butterflies each; shared memory, not
    // threads, limits the CTAs per SM: the fewest rounds, then the fewest threads
    double least = 1e300;
    for (int th = 192; th <= pruned_threads(0); th += 32) {
      double t = 0.0;
      for (int i = 0; i < c.qplan.nst; i++) {
        const int R = c.qplan.st[i].R, items = a.n / R * a.NU;
        t += (double)((items + th - 1) / th) * (30.0 + 8.0 * R);
      }
      if (t < least) {
        least = t;
        threads = th;
      }
    }
  }
  if (c.pairs_per_cta > 0) {
    a.per_cta = (c.pairs_per_cta + a.NU - 1) / a.NU * a.NU;
  } else {
    // groups of units one CTA takes in turn (its weights serve them all): as
    // many as leave the GPU four waves of four CTAs per SM
    const long long groups = (long long)((a.npairs + a.NU - 1) / a.NU) * a.H;
    a.per_cta = a.NU * (int)std::max<long long>(1, std::min<long long>(16, groups / (148 * 16)));
  }
  a.pdiv = make_fastdiv((uint32_t)a.P);
  a.boxdiv = make_fastdiv((uint32_t)a.box);
  a.qdiv = make_fastdiv((uint32_t)a.Q);
  return dispatch_pruned(a, qt, smem, dim3((a.npairs + a.per_cta - 1) / a.per_cta, a.H), threads, st);
}

}  // namespace mc
