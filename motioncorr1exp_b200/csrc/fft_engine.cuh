// Complex helpers, small butterflies and the plan of a mixed-radix transform
// (mixed_fft.cuh runs it).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "f2ops.cuh"
#include "dft_gen.cuh"

namespace mc {

constexpr int kMaxStages = 14;

// q = x / d, r = x % d for x < 2^22 using a float reciprocal plus one fix-up.
struct FastDiv {
  uint32_t d;
  float inv;
};

__host__ __device__ inline FastDiv make_fastdiv(uint32_t d) {
  FastDiv f;
  f.d = d;
  f.inv = 1.0f / (float)d;
  return f;
}

__device__ __forceinline__ void fdivmod(uint32_t x, FastDiv f, uint32_t& q, uint32_t& r) {
  uint32_t qq = (uint32_t)((float)x * f.inv);
  int rr = (int)x - (int)(qq * f.d);
  if (rr < 0) {
    qq -= 1;
    rr += (int)f.d;
  } else if (rr >= (int)f.d) {
    qq += 1;
    rr -= (int)f.d;
  }
  q = qq;
  r = (uint32_t)rr;
}

// One pass of a mixed-radix transform: two neighbouring stages of radix R1, R2
// held in registers (kind R1 * 16 + R2, R2 = 1 for one stage), or one stage of
// a prime above 13.
constexpr int kStageDirect = 1, kStageSymmetric = 2, kStageGeneric = 3;
constexpr int kPrimePairs = 6;  // output pairs a thread forms in the symmetric stage
#define MC_FUSED_LIST(X) \
  X(5, 5) X(7, 3) X(5, 3) X(3, 3) X(11, 2) X(7, 2) X(5, 2) X(3, 2) X(5, 4) X(3, 4) X(3, 8) X(4, 4) X(8, 2)
struct FftStage {
  int kind;
  int R;          // radix (R1 * R2)
  int Ns;         // span before this pass
  int tw, tw2;    // offsets of the factors in the table memory: W_(Ns R1)^(r jm), [(r - 1) * Ns + jm], and the
                  // second stage's W_(Ns R)^(r m), [(r - 1) * Ns * R1 + m]
  int ct, ctp;    // prime stages: offset of the table (float2) and its row pitch (float4): direct
                  // [r][k] = W_p^(r k), symmetric [r - 1][k - 1] = (cos, sin)(2 pi r k / p)
  FastDiv nsdiv;  // divide by Ns
  FastDiv nqdiv;  // divide by n/R
};

struct FftPlan1D {
  int n;
  int nst;
  int ntab;       // float2 entries of the table memory (fft_tables)
  FftStage st[kMaxStages];
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// -i*z (forward) or +i*z (inverse)
template <bool INV>
__device__ __forceinline__ float2 rot90(float2 z) {
  return INV ? make_float2(-z.y, z.x) : make_float2(z.y, -z.x);
}

template <bool INV>
__device__ __forceinline__ void dft_r2(float2* v) {
  float2 a = v[0], b = v[1];
  v[0] = padd(a, b);
  v[1] = psub(a, b);
}

template <bool INV>
__device__ __forceinline__ void dft_r4(float2* v) {
  float2 t0 = padd(v[0], v[2]), t1 = psub(v[0], v[2]);
  float2 t2 = padd(v[1], v[3]), t3 = rot90<INV>(psub(v[1], v[3]));
  v[0] = padd(t0, t2);
  v[2] = psub(t0, t2);
  v[1] = padd(t1, t3);
  v[3] = psub(t1, t3);
}

template <bool INV>
__device__ __forceinline__ void dft_r8(float2* v) {
  const float h = 0.70710678118654752f;
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  dft_r4<INV>(e);
  dft_r4<INV>(o);
  // o[k] *= W8^k
  o[1] = INV ? make_float2(h * (o[1].x - o[1].y), h * (o[1].x + o[1].y))
             : make_float2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
  o[2] = rot90<INV>(o[2]);
  o[3] = INV ? make_float2(-h * (o[3].x + o[3].y), h * (o[3].x - o[3].y))
             : make_float2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[k] = padd(e[k], o[k]);
    v[k + 4] = psub(e[k], o[k]);
  }
}

template <int R, bool INV>
__device__ __forceinline__ void dft_any(float2* v) {
  if constexpr (R == 2) dft_r2<INV>(v);
  else if constexpr (R == 4) dft_r4<INV>(v);
  else if constexpr (R == 8) dft_r8<INV>(v);
  else if constexpr (R == 3) dft_r3<INV>(v);
  else if constexpr (R == 5) dft_r5<INV>(v);
  else if constexpr (R == 7) dft_r7<INV>(v);
  else if constexpr (R == 11) dft_r11<INV>(v);
  else if constexpr (R == 13) dft_r13<INV>(v);
}

}  // namespace mc
