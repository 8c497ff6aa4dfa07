// Pieces of the closure MLP shared by its own kernels (closure_mlp.cu) and by the direct pass that
// evaluates it in place (fused.cu): sizes and parameter offsets, the input / output scaling, the GELU
// with its erf approximation, and the staging of BF16 operands in the canonical K-major layout of
// tcgen05.mma (tcgen05.cuh).  No counterpart in the reference: CRUNA has no learned component.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "../../include/cruna_b200.h"
#include "tcgen05.cuh"

namespace cruna {
namespace mlp {

constexpr int IN = 12, HID = 64, OUT = 6;
constexpr int OW1 = 0, OB1 = OW1 + HID * IN, OW2 = OB1 + HID, OB2 = OW2 + HID * HID, OW3 = OB2 + HID,
              OB3 = OW3 + OUT * HID, NPARAMS = OB3 + OUT;
static_assert(NPARAMS == CRUNA_MLP_NPARAMS, "parameter count");
constexpr long long kWaitLimit = 1LL << 22;  // mbarrier polls before a kernel gives up (error flag)

struct Scaling {
  float in_mean[IN];
  float in_inv[IN];   // 1 / in_scale
  float out_scale[OUT];
};

// erf by the rational approximation of Abramowitz & Stegun, Handbook of Mathematical Functions, 7.1.26
// (|error| <= 1.5e-7, far below the BF16 rounding of the activations), with fast reciprocal and
// exponential; e2 returns exp(-x^2) for the GELU derivative.  The activations cost most of the
// forward kernel's instructions, so this replaces erff.
__device__ __forceinline__ float erf_as(float x, float &e2) {
  const float ax = fabsf(x);
  const float t = __fdividef(1.0f, fmaf(0.3275911f, ax, 1.0f));
  float p = fmaf(1.061405429f, t, -1.453152027f);
  p = fmaf(p, t, 1.421413741f);
  p = fmaf(p, t, -0.284496736f);
  p = fmaf(p, t, 0.254829592f);
  e2 = __expf(-ax * ax);
  return copysignf(1.0f - p * t * e2, x);
}

// GELU (erf form) z Phi(z) = 0.5 z (1 + erf(z / sqrt 2)) and its derivative Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_and_grad(float z, float &grad) {
  float e2;  // exp(-z^2 / 2)
  const float cdf = 0.5f * (1.0f + erf_as(z * 0.70710678118654752f, e2));
  grad = cdf + z * e2 * 0.39894228040143268f;
  return z * cdf;
}

// Two GELUs at once on packed FP32 arithmetic (fma.rn.f32x2 issues two lanes' operations as one): with
// Phi(-|z|) = h, gelu(z) = max(z, 0) - |z| h, and h = (P(t) / 2) t exp(-z^2 / 2) from the same approximation
// as erf_as (t = 1 / (1 + 0.3275911 |z| / sqrt 2), one half folded into P's coefficients).  15 issue slots and 4
// special-function operations a pair, against about 44 and 4 one at a time.
__device__ __forceinline__ uint64_t f2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_split(uint64_t v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void gelu2(uint64_t z, float &ga, float &gb) {
  float za, zb, da, db, sa, sb;
  f2_split(z, za, zb);
  // -|z|, held at -30 where h is exactly zero, so that an infinite activation stays infinite (not inf * 0)
  const uint64_t nz = f2(fmaxf(-fabsf(za), -30.0f), fmaxf(-fabsf(zb), -30.0f));
  f2_split(fma2(nz, f2(-0.23164189f, -0.23164189f), f2(1.0f, 1.0f)), da, db);  // 1 + 0.3275911 |z| / sqrt 2
  const uint64_t t = f2(rcp_approx(da), rcp_approx(db));
  f2_split(mul2(mul2(z, f2(-0.72134752f, -0.72134752f)), z), sa, sb);          // -z^2 / (2 ln 2)
  const uint64_t e = f2(ex2_approx(sa), ex2_approx(sb));
  uint64_t p = fma2(f2(0.5307027145f, 0.5307027145f), t, f2(-0.7265760135f, -0.7265760135f));
  p = fma2(p, t, f2(0.7107068705f, 0.7107068705f));
  p = fma2(p, t, f2(-0.142248368f, -0.142248368f));
  p = fma2(p, t, f2(0.127414796f, 0.127414796f));
  const uint64_t h = mul2(mul2(p, t), e);
  f2_split(fma2(nz, h, f2(fmaxf(za, 0.0f), fmaxf(zb, 0.0f))), ga, gb);
}

// v[i] = gelu(v[i] + b[i]), 16 values; b in shared memory (8-byte aligned)
__device__ __forceinline__ void gelu16(float *v, const float *b) {
  const uint64_t *b2 = reinterpret_cast<const uint64_t *>(b);
#pragma unroll
  for (int i = 0; i < 8; ++i) gelu2(add2(f2(v[2 * i], v[2 * i + 1]), b2[i]), v[2 * i], v[2 * i + 1]);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);  // .x = a (low half), .y = b
  return *reinterpret_cast<uint32_t *>(&h);
}

// 8 consecutive row elements (k0 .. k0+7, k0 % 8 == 0) of row r of an R x K tile
__device__ __forceinline__ void put8(__nv_bfloat16 *tile, int r, int k0, int K, const float *v) {
  uint4 u;
  u.x = pack2(v[0], v[1]);
  u.y = pack2(v[2], v[3]);
  u.z = pack2(v[4], v[5]);
  u.w = pack2(v[6], v[7]);
  *reinterpret_cast<uint4 *>(tile + tc::kmaj(r, k0, K)) = u;
}

// stage weights as B operands ([N][K], K-major); transposed copies for the backward products
__device__ inline void stage_weights(const float *__restrict__ P, __nv_bfloat16 *W1, __nv_bfloat16 *W2, __nv_bfloat16 *W3,
                              __nv_bfloat16 *W3T, __nv_bfloat16 *W2T) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < HID * 16; i += nt) {
    const int r = i >> 4, k = i & 15;
    W1[tc::kmaj(r, k, 16)] = __float2bfloat16_rn(k < IN ? P[OW1 + r * IN + k] : 0.0f);
  }
  for (int i = tid; i < HID * HID; i += nt) {
    const int r = i >> 6, k = i & 63;
    W2[tc::kmaj(r, k, 64)] = __float2bfloat16_rn(P[OW2 + r * HID + k]);
    if (W2T) W2T[tc::kmaj(k, r, 64)] = __float2bfloat16_rn(P[OW2 + r * HID + k]);
  }
  for (int i = tid; i < 16 * HID; i += nt) {
    const int r = i >> 6, k = i & 63;
    const float w = r < OUT ? P[OW3 + r * HID + k] : 0.0f;
    W3[tc::kmaj(r, k, 64)] = __float2bfloat16_rn(w);
    if (W3T) W3T[tc::kmaj(k, r, 16)] = __float2bfloat16_rn(w);  // [64][16]: (j, o) = W3[o][j]
  }
}

}  // namespace mlp

// device parameters, scaling and error flag of a network (closure_mlp.cu), for kernels that evaluate
// it in place
void mlp_device_view(struct cruna_mlp *h, const float **P, mlp::Scaling *sc, int **flag);

}  // namespace cruna
