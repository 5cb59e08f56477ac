// Mixed-radix Stockham FFT over shared memory, for any length without a
// compiled two-level split.
//
// A transform of length n runs as a list of stages with radices R_0..R_{s-1}
// (product n).  Stage s with span Ns = R_0*..*R_{s-1} does, for every
// butterfly j in [0, n/R):
//     v[r]  = src[j + r*n/R] * W_(Ns R)^(r * (j mod Ns))          (r >= 1)
//     v     = DFT_R(v)
//     dst[(j div Ns)*Ns*R + (j mod Ns) + r*Ns] = v[r]
// which leaves the result in natural order (autosort) after the last stage.
// W_n = exp(-2 pi i / n) for the forward transform, its conjugate for the
// inverse; both transforms are un-normalised (cuFFT / FFTW convention).
//
// A batch of B transforms shares the stages.  Two element layouts exist:
//   rows        element (b, i) at b*ld + i   (thread index: i fastest)
//   interleaved element (b, i) at b + B*i    (thread index: b fastest)
// Both keep consecutive threads on consecutive shared-memory words.
//
// What bounds a stage is its shared-memory and twiddle traffic, not its
// arithmetic, so two neighbouring stages R1, R2 run as one pass where R1 * R2
// values fit a thread's registers (fused below: the same operations on the same
// factors in the same order, so the transform's bits do not depend on what is
// fused); the first pass reads its input through `ldf` (global memory or a
// staged row) and the last hands its output to `stf`, which saves a trip
// through shared memory at either end; a stage's twiddles lie in global memory
// in the order its threads read them.  Odd radices come first: a first stage of
// even radix R writes with stride R, gcd(R, 16) lanes to a bank pair.
//
// Measured per frame, row / column pass, before (one stage a pass, three shared
// buffers with the tables copied in, one output of a prime's direct sum a
// thread) and now: 4092^2 = 31 | 11 | 3 x 4 605 / 520 -> 182 / 173 us; 1500^2 =
// 5 x 5 | 5 x 3 | 4 55 / 41 -> 13.5 / 10.0 us; 520^2 = 13 | 5 | 8 (30 frames)
// 13.6 / 13.9 -> 2.0 / 1.5 us.  Powers of two and 3710 keep the two-level form
// (kcommon.cuh), which has one exchange instead of two.
#pragma once
#include "fft_engine.cuh"

namespace mc {

// Butterfly index t of a batch stage -> (transform b, butterfly j).
template <bool INTERLEAVED>
__device__ __forceinline__ void bfly_index(uint32_t t, const FftStage& s, FastDiv bdiv, uint32_t& b, uint32_t& j) {
  if (INTERLEAVED) fdivmod(t, bdiv, j, b);
  else fdivmod(t, s.nqdiv, b, j);
}

// Stages of radix R1 and R2 (R2 = 1: one stage) in one pass over B transforms.
// With R = R1 R2, thread j holds x[j + i n/R], i = r2 + R2 r1: for every r2 the
// radix-R1 butterfly j + r2 n/R of the first stage, whose outputs r1 are the
// inputs r2 of the second stage's butterfly (j div Ns) Ns R1 + jm + r1 Ns.
template <int R1, int R2, bool INV, bool INTERLEAVED, class Ld, class St>
__device__ __forceinline__ void stage_fused(const float2* src, float2* dst, const FftStage& s, int B, FastDiv bdiv,
                                            int ld, const float2* __restrict__ tw, int tid, int nth, bool first,
                                            bool last, Ld&& ldf, St&& stf) {
  constexpr int R = R1 * R2;
  const int nq = (int)s.nqdiv.d, Ns = s.Ns;
  const int total = nq * B;
  auto factor = [&](const float2* w) {
    float2 f = __ldg(w);
    if (INV) f.y = -f.y;
    return f;
  };
  for (int t = tid; t < total; t += nth) {
    uint32_t j, b, jq, jm = 0;
    bfly_index<INTERLEAVED>((uint32_t)t, s, bdiv, b, j);
    float2 v[R2][R1];
    if (first) {
      jq = j;
#pragma unroll
      for (int i = 0; i < R; i++) v[i % R2][i / R2] = ldf((int)b, (int)j + i * nq);
    } else {
      fdivmod(j, s.nsdiv, jq, jm);
      const float2* w = tw + s.tw + jm;
#pragma unroll
      for (int r1 = 0; r1 < R1; r1++) {
        float2 f;
        if (r1) f = factor(w + (r1 - 1) * Ns);
#pragma unroll
        for (int r2 = 0; r2 < R2; r2++) {
          const int i = (int)j + (r2 + R2 * r1) * nq;
          const float2 x = INTERLEAVED ? src[b + B * i] : src[b * ld + i];
          v[r2][r1] = r1 ? cmul(x, f) : x;
        }
      }
    }
#pragma unroll
    for (int r2 = 0; r2 < R2; r2++) dft_any<R1, INV>(v[r2]);
    const int base = (int)jq * Ns * R + (int)jm;
    auto put = [&](int i, float2 x) {
      if (last) stf(dst, (int)b, i, x);
      else dst[INTERLEAVED ? b + B * i : b * ld + i] = x;
    };
    if constexpr (R2 == 1) {
#pragma unroll
      for (int r1 = 0; r1 < R1; r1++) put(base + r1 * Ns, v[0][r1]);
    } else {
      const float2* w = tw + s.tw2 + jm;
#pragma unroll
      for (int r1 = 0; r1 < R1; r1++) {
        float2 u[R2];
        u[0] = v[0][r1];
#pragma unroll
        for (int r2 = 1; r2 < R2; r2++) u[r2] = cmul(v[r2][r1], factor(w + ((r2 - 1) * R1 + r1) * Ns));
        dft_any<R2, INV>(u);
#pragma unroll
        for (int r2 = 0; r2 < R2; r2++) put(base + (r1 + r2 * R1) * Ns, u[r2]);
      }
    }
  }
}

// Prime radix p (17..127) as the first stage (a second such prime, or a larger
// one, takes stage_generic), every output the direct sum
//   X_k = sum_r x_r W_p^(r k), r ascending.
// A thread forms G outputs of one butterfly, so an input read serves G outputs
// and the factors (the same for all threads of a warp) come two to a 16-byte
// load from the table [r][k].
template <bool INV, bool INTERLEAVED, class Ld, class St>
__device__ __forceinline__ void stage_direct(float2* cur, float2* dst, const FftStage& s, int B, FastDiv bdiv, int ld,
                                             const float2* __restrict__ tw, int tid, int nth, bool last, Ld&& ldf,
                                             St&& stf) {
  constexpr int G = 8;
  const int p = s.R, nq = (int)s.nqdiv.d, nb = nq * B, ng = (p + G - 1) / G;
  const FastDiv nbdiv = make_fastdiv((uint32_t)nb);
  for (int t = tid; t < nb * p; t += nth) {
    uint32_t r, jb, j, b;
    fdivmod((uint32_t)t, nbdiv, r, jb);
    bfly_index<INTERLEAVED>(jb, s, bdiv, b, j);
    const int i = (int)j + (int)r * nq;
    cur[INTERLEAVED ? b + B * i : b * ld + i] = ldf((int)b, i);
  }
  __syncthreads();
  const float4* __restrict__ tab = reinterpret_cast<const float4*>(tw + s.ct);
  for (int t = tid; t < nb * ng; t += nth) {
    uint32_t g, jb, j, b;
    fdivmod((uint32_t)t, nbdiv, g, jb);
    bfly_index<INTERLEAVED>(jb, s, bdiv, b, j);
    const int step = INTERLEAVED ? B * nq : nq;
    const float2* x = cur + (INTERLEAVED ? b + B * j : b * ld + j);
    float2 A[G];
#pragma unroll
    for (int i = 0; i < G; i++) A[i] = x[0];
    const float4* tr = tab + s.ctp + (int)g * (G / 2);
    for (int r = 1; r < p; r++) {
      x += step;
      const float2 a = *x;
#pragma unroll
      for (int i = 0; i < G / 2; i++) {
        const float4 c = __ldg(tr + i);
        const float2 u = cmul(a, make_float2(c.x, INV ? -c.y : c.y)), v = cmul(a, make_float2(c.z, INV ? -c.w : c.w));
        A[2 * i] = cadd(A[2 * i], u);
        A[2 * i + 1] = cadd(A[2 * i + 1], v);
      }
      tr += s.ctp;
    }
#pragma unroll
    for (int i = 0; i < G; i++) {
      const int k = (int)g * G + i;
      if (k >= p) break;
      const int o = (int)j * p + k;  // span 1
      if (last) stf(dst, (int)b, o, A[i]);
      else dst[INTERLEAVED ? b + B * o : b * ld + o] = A[i];
    }
  }
}

// Radix 53 in the symmetric direct form: with a_r = x_r + x_{p-r},
// b_r = x_r - x_{p-r}, r = 1..h = (p-1)/2,
//   A_k = x_0 + sum_r a_r cos(2 pi r k / p),  B_k = sum_r b_r sin(2 pi r k / p)
//   X_k, X_{p-k} = A_k -/+ i B_k  (forward; inverse the other way round)
// The a and b replace the inputs in place (every thread its own two elements);
// then a thread forms G output pairs of one butterfly, so each a_r, b_r read
// from shared memory serves G pairs, and the cosines and sines (the same for
// all threads of a warp) come two pairs to a 16-byte load.
template <int G, bool INV, bool INTERLEAVED, class St>
__device__ __forceinline__ void symmetric_outputs(const float2* cur, float2* dst, const FftStage& s, int B, FastDiv bdiv,
                                              int ld, const float2* __restrict__ tw, int tid, int nth, bool last,
                                              St&& stf) {
  const int p = s.R, h = (p - 1) / 2, nq = (int)s.nqdiv.d, Ns = s.Ns;
  const int nb = nq * B, ng = (h + G - 1) / G;
  const float4* __restrict__ tab = reinterpret_cast<const float4*>(tw + s.ct);
  const FastDiv nbdiv = make_fastdiv((uint32_t)nb);
  for (int t = tid; t < nb * ng; t += nth) {
    uint32_t g, jb, j, b, jq, jm;
    fdivmod((uint32_t)t, nbdiv, g, jb);
    bfly_index<INTERLEAVED>(jb, s, bdiv, b, j);
    fdivmod(j, s.nsdiv, jq, jm);
    const int step = INTERLEAVED ? B * nq : nq;
    const float2* x = cur + (INTERLEAVED ? b + B * j : b * ld + j);
    const float2 x0 = x[0];
    float2 A[G], S[G], sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < G; i++) {
      A[i] = x0;
      S[i] = make_float2(0.f, 0.f);
    }
    const float4* tr = tab + (int)g * (G / 2);
    const float2* xa = x + step;
    const float2* xb = x + (p - 1) * step;
    for (int r = 0; r < h; r++) {
      const float2 a = *xa, d = *xb;
      sum = r ? cadd(sum, a) : a;
#pragma unroll
      for (int i = 0; i < G / 2; i++) {
        const float4 c = __ldg(tr + i);
        A[2 * i].x = fmaf(a.x, c.x, A[2 * i].x);
        A[2 * i].y = fmaf(a.y, c.x, A[2 * i].y);
        S[2 * i].x = fmaf(d.x, c.y, S[2 * i].x);
        S[2 * i].y = fmaf(d.y, c.y, S[2 * i].y);
        A[2 * i + 1].x = fmaf(a.x, c.z, A[2 * i + 1].x);
        A[2 * i + 1].y = fmaf(a.y, c.z, A[2 * i + 1].y);
        S[2 * i + 1].x = fmaf(d.x, c.w, S[2 * i + 1].x);
        S[2 * i + 1].y = fmaf(d.y, c.w, S[2 * i + 1].y);
      }
      xa += step;
      xb -= step;
      tr += s.ctp;
    }
    const int base = (int)jq * Ns * p + (int)jm;
    auto put = [&](int k, float2 v) {
      const int i = base + k * Ns;
      if (last) stf(dst, (int)b, i, v);
      else dst[INTERLEAVED ? b + B * i : b * ld + i] = v;
    };
    if (g == 0) put(0, cadd(x0, sum));
#pragma unroll
    for (int i = 0; i < G; i++) {
      const int k = (int)g * G + i + 1;
      if (k <= h) {
        const float2 lo = make_float2(A[i].x + S[i].y, A[i].y - S[i].x);
        const float2 hi = make_float2(A[i].x - S[i].y, A[i].y + S[i].x);
        put(k, INV ? hi : lo);
        put(p - k, INV ? lo : hi);
      }
    }
  }
}

template <bool INV, bool INTERLEAVED, class Ld, class St>
__device__ __forceinline__ void stage_symmetric(float2* cur, float2* dst, const FftStage& s, int B, FastDiv bdiv, int ld,
                                            const float2* __restrict__ tw, int tid, int nth, bool first, bool last,
                                            Ld&& ldf, St&& stf) {
  const int p = s.R, h = (p - 1) / 2, nq = (int)s.nqdiv.d, Ns = s.Ns, nb = nq * B;
  const FastDiv nbdiv = make_fastdiv((uint32_t)nb);
  for (int t = tid; t < nb * (h + 1); t += nth) {
    uint32_t r, jb, j, b, jq, jm;
    fdivmod((uint32_t)t, nbdiv, r, jb);
    bfly_index<INTERLEAVED>(jb, s, bdiv, b, j);
    const int i0 = (int)j + (int)r * nq, i1 = (int)j + (p - (int)r) * nq;
    float2* x0 = cur + (INTERLEAVED ? b + B * i0 : b * ld + i0);
    if (r == 0) {
      if (first) *x0 = ldf((int)b, i0);
      continue;
    }
    float2* x1 = cur + (INTERLEAVED ? b + B * i1 : b * ld + i1);
    float2 u, v;
    if (first) {
      u = ldf((int)b, i0);
      v = ldf((int)b, i1);
    } else {
      fdivmod(j, s.nsdiv, jq, jm);
      float2 f = __ldg(tw + s.tw + ((int)r - 1) * Ns + jm), e = __ldg(tw + s.tw + (p - (int)r - 1) * Ns + jm);
      if (INV) {
        f.y = -f.y;
        e.y = -e.y;
      }
      u = cmul(*x0, f);
      v = cmul(*x1, e);
    }
    *x0 = cadd(u, v);
    *x1 = csub(u, v);
  }
  __syncthreads();
  symmetric_outputs<kPrimePairs, INV, INTERLEAVED>(cur, dst, s, B, bdiv, ld, tw, tid, nth, last, stf);
}

// Other primes, and a table prime that is not the first stage: every output of
// every butterfly as a direct sum,
//   X_k = sum_r src[j + r*n/R] * W_n^(r*((j mod Ns)*tws + k*n/R)).
template <bool INV, bool INTERLEAVED, class Ld, class St>
__device__ void stage_generic(float2* src, float2* dst, const FftStage& s, int n, int B, FastDiv bdiv, int ld,
                              const float2* __restrict__ tw, int tid, int nth, bool first, bool last, Ld&& ldf,
                              St&& stf) {
  const int R = s.R;
  const int nq = (int)s.nqdiv.d;
  if (first) {
    const FastDiv ndiv = make_fastdiv((uint32_t)n);
    for (int t = tid; t < n * B; t += nth) {
      uint32_t b, i;
      if (INTERLEAVED) fdivmod((uint32_t)t, bdiv, i, b);
      else fdivmod((uint32_t)t, ndiv, b, i);
      src[INTERLEAVED ? b + B * i : b * ld + i] = ldf((int)b, (int)i);
    }
    __syncthreads();
  }
  const int total = nq * B * R;
  const FastDiv rdiv = make_fastdiv((uint32_t)R);
  for (int t = tid; t < total; t += nth) {
    uint32_t jb, k, j, b, jq, jm;
    fdivmod((uint32_t)t, rdiv, jb, k);
    bfly_index<INTERLEAVED>(jb, s, bdiv, b, j);
    fdivmod(j, s.nsdiv, jq, jm);
    const int step = ((int)jm * (nq / s.Ns) + (int)k * nq) % n;
    int e = 0;
    float2 acc = make_float2(0.f, 0.f);
    for (int r = 0; r < R; r++) {
      const int i = (int)j + r * nq;
      const float2 x = INTERLEAVED ? src[b + B * i] : src[b * ld + i];
      float2 w = __ldg(tw + e);
      if (INV) w.y = -w.y;
      const float2 p = cmul(x, w);
      acc.x += p.x;
      acc.y += p.y;
      e += step;
      if (e >= n) e -= n;
    }
    const int i = (int)jq * s.Ns * R + (int)jm + (int)k * s.Ns;
    if (last) stf(dst, (int)b, i, acc);
    else dst[INTERLEAVED ? b + B * i : b * ld + i] = acc;
  }
}

// Runs all stages.  ldf(b, i) gives input element i of transform b; the last
// stage hands element i to stf(dst, b, i, value), dst being the buffer no
// thread reads any more.  Input staged in s1 (ldf reading s1) is read before
// anything else is written there.  No barrier after the last stage.
template <bool INV, bool INTERLEAVED, class Ld, class St>
__device__ __forceinline__ void fft_exec(float2* s0, float2* s1, const FftPlan1D& p, int B, int ld,
                                         const float2* __restrict__ tw, int tid, int nth, Ld&& ldf, St&& stf) {
  const FastDiv bdiv = make_fastdiv((uint32_t)B);
  float2 *cur = s1, *nxt = s0;
  if (p.nst == 0)  // length 1
    for (int t = tid; t < B; t += nth) stf(s0, t, 0, ldf(t, 0));
  for (int si = 0; si < p.nst; si++) {
    const FftStage& s = p.st[si];
    const bool first = si == 0, last = si == p.nst - 1;
#define MC_RADIX(A, B2)                                                                                         \
  case A * 16 + B2:                                                                                             \
    stage_fused<A, B2, INV, INTERLEAVED>(cur, nxt, s, B, bdiv, ld, tw, tid, nth, first, last, ldf, stf);        \
    break;
    switch (s.kind) {
      MC_RADIX(2, 1) MC_RADIX(3, 1) MC_RADIX(4, 1) MC_RADIX(5, 1) MC_RADIX(7, 1) MC_RADIX(8, 1) MC_RADIX(11, 1)
      MC_RADIX(13, 1)
      MC_FUSED_LIST(MC_RADIX)
      case kStageDirect: stage_direct<INV, INTERLEAVED>(cur, nxt, s, B, bdiv, ld, tw, tid, nth, last, ldf, stf); break;
      case kStageSymmetric:
        stage_symmetric<INV, INTERLEAVED>(cur, nxt, s, B, bdiv, ld, tw, tid, nth, first, last, ldf, stf);
        break;
      default:
        stage_generic<INV, INTERLEAVED>(cur, nxt, s, p.n, B, bdiv, ld, tw, tid, nth, first, last, ldf, stf);
    }
#undef MC_RADIX
    if (!last) __syncthreads();
    float2* t = cur;
    cur = nxt;
    nxt = t;
  }
}

}  // namespace mc
