// The NVFP4 encoding of one 16-element block (see quantize.cu for the contract), shared by the quantiser and by the decode
// front end.
#pragma once
#include "kernels.cuh"
#include "ptx.cuh"

namespace b200 {

// RN(a / b) from r = RN(1 / b): Markstein's residual correction, twice. The first step brings the quotient within an ulp, the
// second (whose residual is then exact in one fma) rounds it correctly.
DEV float div_rn(float a, float b, float r) {
  float q = __fmul_rn(a, r);
  q = __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// One block of 16 bf16 values (eight words) -> its E4M3 scale byte and 16 E2M1 codes.
//
// Quotients x / (stored * gs) without sixteen IEEE divisions per block. With r = RN(1 / d), q0 = RN(x * r), the residual
// rem = x - q0 * d is exact in one fma (q0 is within 1.5 ulp of x / d and x has only 8 significant bits), and
// q1 = RN(q0 + rem * r) is the correctly rounded quotient (Markstein's residual correction with a correctly rounded
// reciprocal). The E2M1 code only depends on the side of seven thresholds the quotient lies on, so a last-bit error could
// matter only when x / d is within an ulp of a threshold; the test suite sweeps every bf16 value against every E4M3 scale x a
// set of global scales and compares the codes with true division. The chain runs on -x and -r: -rem = q0 * d + (-x) and
// q1 = (-rem) * (-r) + q0 round alike, and both zeros come out with the sign of x (they encode as 0 and 8).
// EXACT_DIV selects IEEE division instead (global scales so small or large that the residual could leave the normal range).
template <bool EXACT_DIV>
DEV uint32_t quantize_block(const uint32_t (&w)[8], float gs, float rgs, uint32_t (&packed)[2]) {
  __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));      // the largest magnitude, exact in bf16
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
  float peak = fmaxf(__low2float(m), __high2float(m));
  peak = fmaxf(peak, 9.5367431640625e-07f);                       // clamp_min(2^-20), before the global scale
  float scale;
  if (EXACT_DIV) {
    scale = __fdiv_rn(peak, 6.0f);
    if (gs != 1.0f) scale = __fdiv_rn(scale, gs);
  } else {
    // a peak beyond 6144 * gs only ever gives a scale that the clamp below turns into 448
    scale = div_rn(fminf(peak, 6144.0f * gs), 6.0f, 1.0f / 6.0f);
    scale = div_rn(scale, gs, rgs);
  }
  scale = fminf(fmaxf(scale, 0.001953125f), 448.0f);               // clamp(2^-9, 448)
  const uint32_t sbyte = cvt_e4m3(scale);
  const float d = __fmul_rn(e4m3_to_f32(sbyte), gs);               // the reference divides by stored * gs
  const float nr = EXACT_DIV ? 0.f : -__frcp_rn(d);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float q[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t u = w[4 * h + i];
      if (EXACT_DIV) {
        q[2 * i] = __fdiv_rn(__uint_as_float(u << 16), d);
        q[2 * i + 1] = __fdiv_rn(__uint_as_float(u & 0xFFFF0000u), d);
      } else {
        const float2 nx = make_float2(__uint_as_float(u * 65536u + 0x80000000u), __uint_as_float((u & 0xFFFF0000u) ^ 0x80000000u));
        const float2 nr2 = make_float2(nr, nr), q0 = mul2(nx, nr2), q1 = fma2(fma2(q0, make_float2(d, d), nx), nr2, q0);
        q[2 * i] = q1.x;
        q[2 * i + 1] = q1.y;
      }
    }
    packed[h] = cvt_e2m1x8(q);
  }
  return sbyte;
}

// stored * gs stays a normal number with room for the residual of a bf16 numerator inside 2^-40 .. 2^40
inline bool quantize_fast(float gs) { return gs >= 0x1p-40f && gs <= 0x1p40f; }

}  // namespace b200
