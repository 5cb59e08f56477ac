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
// arithmetic, so the plan takes few stages of large radix (up to 16, in
// registers); the first stage reads its input through `ldf` (global memory or
// a staged row) and the last hands its output to `stf`, which saves a pass
// over shared memory at either end; a stage's twiddles lie in global memory in
// the order its threads read them.  Odd radices come first: a first stage of
// even radix R would write with stride R, gcd(R, 16) lanes to a bank pair.
//
// Measured per frame, row / column pass, before (radices up to 13, a direct sum
// per output for other primes, tables copied to shared memory) and now:
// 4092^2 = 31 x 12 x 11 605 / 520 -> 130 / 104 us; 1500^2 = 15 x 10 x 10 55 /
// 41 -> 14 / 7.5 us; 520^2 (30 frames) 13.6 / 13.9 -> 2.1 / 1.5 us.  Powers of
// two and 3710 keep the two-level form (kcommon.cuh), which has one exchange
// instead of two: 4096^2 84 / 44 us against 129 / 69 here.
#pragma once
#include "codelets_gen.cuh"
#include "fft_engine.cuh"

namespace mc {

template <int R, bool INV>
__device__ __forceinline__ void radix_bfly(float2* v) {
  if constexpr (R == 9 || R == 16) fft_reg<R, INV>(v);
  else if constexpr (R == 6 || R == 10 || R == 12 || R == 14 || R == 15) fft_reg_pf<R, INV>(v);
  else dft_any<R, INV>(v);
}

// Butterfly index t of a batch stage -> (transform b, butterfly j).
template <bool INTERLEAVED>
__device__ __forceinline__ void bfly_index(uint32_t t, const FftStage& s, FastDiv bdiv, uint32_t& b, uint32_t& j) {
  if (INTERLEAVED) fdivmod(t, bdiv, j, b);
  else fdivmod(t, s.nqdiv, b, j);
}

// One stage of compile-time radix R over B transforms.
template <int R, bool INV, bool INTERLEAVED, class Ld, class St>
__device__ __forceinline__ void stage_fixed(const float2* src, float2* dst, const FftStage& s, int B, FastDiv bdiv,
                                            int ld, const float2* __restrict__ tw, int tid, int nth, bool first,
                                            bool last, Ld&& ldf, St&& stf) {
  const int nq = (int)s.nqdiv.d, Ns = s.Ns;
  const int total = nq * B;
  for (int t = tid; t < total; t += nth) {
    uint32_t j, b, jq, jm = 0;
    bfly_index<INTERLEAVED>((uint32_t)t, s, bdiv, b, j);
    float2 v[R];
    if (first) {
      jq = j;
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = ldf((int)b, (int)j + r * nq);
    } else {
      fdivmod(j, s.nsdiv, jq, jm);
      const float2* w = tw + s.tw + jm;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int i = (int)j + r * nq;
        v[r] = INTERLEAVED ? src[b + B * i] : src[b * ld + i];
        if (r) {
          float2 f = __ldg(w + (r - 1) * Ns);
          if (INV) f.y = -f.y;
          v[r] = cmul(v[r], f);
        }
      }
    }
    radix_bfly<R, INV>(v);
    const int base = (int)jq * Ns * R + (int)jm;
    if (last) {
#pragma unroll
      for (int r = 0; r < R; r++) stf(dst, (int)b, base + r * Ns, v[r]);
    } else {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int i = base + r * Ns;
        dst[INTERLEAVED ? b + B * i : b * ld + i] = v[r];
      }
    }
  }
}

// Radix-p stage for a prime p with a table (17..127), in the symmetric direct
// form: with a_r = x_r + x_{p-r}, b_r = x_r - x_{p-r}, r = 1..h = (p-1)/2,
//   A_k = x_0 + sum_r a_r cos(2 pi r k / p),  B_k = sum_r b_r sin(2 pi r k / p)
//   X_k, X_{p-k} = A_k -/+ i B_k  (forward; inverse the other way round)
// The a and b replace the inputs in place (every thread its own two elements);
// then a thread forms G output pairs of one butterfly, so each a_r, b_r read
// from shared memory serves G pairs, and the cosines and sines (the same for
// all threads of a warp) come two pairs to a 16-byte load.
template <int G, bool INV, bool INTERLEAVED, class St>
__device__ __forceinline__ void prime_outputs(const float2* cur, float2* dst, const FftStage& s, int B, FastDiv bdiv,
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
    float2 A[G], S[G], sum = x0;
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
      sum = cadd(sum, a);
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
    if (g == 0) put(0, sum);
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
__device__ __forceinline__ void stage_prime(float2* cur, float2* dst, const FftStage& s, int B, FastDiv bdiv, int ld,
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
  if (s.G == 6) prime_outputs<6, INV, INTERLEAVED>(cur, dst, s, B, bdiv, ld, tw, tid, nth, last, stf);
  else prime_outputs<8, INV, INTERLEAVED>(cur, dst, s, B, bdiv, ld, tw, tid, nth, last, stf);
}

// Larger primes: every output of every butterfly as a direct sum,
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
#define MC_RADIX(RR)                                                                                            \
  case RR:                                                                                                      \
    stage_fixed<RR, INV, INTERLEAVED>(cur, nxt, s, B, bdiv, ld, tw, tid, nth, first, last, ldf, stf);           \
    break;
    switch (s.R) {
      MC_RADIX(2) MC_RADIX(3) MC_RADIX(4) MC_RADIX(5) MC_RADIX(6) MC_RADIX(7) MC_RADIX(8) MC_RADIX(9)
      MC_RADIX(10) MC_RADIX(11) MC_RADIX(12) MC_RADIX(13) MC_RADIX(14) MC_RADIX(15) MC_RADIX(16)
      default:
        if (s.G) stage_prime<INV, INTERLEAVED>(cur, nxt, s, B, bdiv, ld, tw, tid, nth, first, last, ldf, stf);
        else stage_generic<INV, INTERLEAVED>(cur, nxt, s, p.n, B, bdiv, ld, tw, tid, nth, first, last, ldf, stf);
    }
#undef MC_RADIX
    if (!last) __syncthreads();
    float2* t = cur;
    cur = nxt;
    nxt = t;
  }
}

}  // namespace mc
