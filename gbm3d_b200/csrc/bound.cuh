// Device code shared by the matchers that bound candidates with f16 warp MMAs
// (match_bound.cu, video_bound.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace gbm3d {

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f16_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// The bound.  All values are centred by a number m0 common to the CTA and
// rounded to f16: x16, w16.  With r = ||x - w|| (the true distance of two patches)
// and r16 = ||x16 - w16||, |r - r16| <= u (||x'|| + ||w'||) + 2 eta
// <= u (2 ||x'|| + r) + 2 eta, u = 2^-11 the f16 rounding unit, eta = side 2^-25 its
// subnormal part: the error is that of two roundings, not of a product, so it
// vanishes with the patch's contrast.  The computed squared distance is
// d = ||x16||^2 - 2 v, v = <x16, w16> - ||w16||^2 / 2 (the norm sums are those of the rounded
// values), with |d - r16^2| <= KAPPA (||x16||^2 + ||w16||^2); KAPPA covers the MMA steps
// (each of a step's nonzero addends truncated at 2^-23 of the largest) and the
// FP32 sums.  The exact distance F of the ranking, a serial FP32 chain, lies
// within a factor 1 +- GAMMA of r^2.
//   T bounds the computed d of at least K candidates, nx = ||x16||^2.  Then the K-th
// smallest F is at most R^2 (1 + GAMMA) below, every candidate of the exact top K
// has r <= R (1 + GAMMA2), and a computed d of at most the value returned.
struct Bound8 {  // 8 x 8 patches: 8 steps of 9 addends; 64-term chains (70 2^-24)
  static constexpr float ETA2 = 4.8e-7f, KAPPA = 2.2e-5f, GAMMA2 = 1.0e-5f;
};
struct Bound32 {  // 32 x 32 patches: 96 steps of at most 17 addends; 1024-term chains (1030 2^-24)
  static constexpr float ETA2 = 1.92e-6f, KAPPA = 2.2e-4f, GAMMA2 = 1.3e-4f;
};
template <class B>
__device__ __forceinline__ float candidate_threshold(float T, float nx) {
  constexpr float U = 4.8852e-4f;  // 2^-11 (1 + 2^-11)
  const float X = sqrtf(nx) * (1.f + 2.f * U) + B::ETA2;                                      // >= ||x'||
  const float A = sqrtf((fmaxf(T, 0.f) + 3.f * B::KAPPA * nx) * (1.f + 3.f * B::KAPPA));      // >= r16 of K candidates
  const float R = (A + 2.f * U * X + B::ETA2) * (1.f + 2.f * U) * (1.f + B::GAMMA2);          // >= r of the exact top K
  const float R16 = R * (1.f + U) + 2.f * U * X + B::ETA2;                                    // >= their r16
  return (R16 * R16 * (1.f + 2.f * B::KAPPA) + 3.f * B::KAPPA * nx) * (1.f + 1e-6f);          // >= their d
}

// Descending bitonic sort of one value per lane.
__device__ __forceinline__ float sort_desc(float v, int lane) {
#pragma unroll
  for (int k2 = 2; k2 <= 32; k2 <<= 1)
#pragma unroll
    for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
      const float o = __shfl_xor_sync(0xffffffffu, v, j2);
      const bool up = ((lane & k2) == 0), lower = ((lane & j2) == 0);
      v = (lower == up) ? fmaxf(v, o) : fminf(v, o);
    }
  return v;
}

}  // namespace gbm3d
