// Exact expansion of NVFP4 weights to bf16, shared by the W4A16 kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "ptx.cuh"

namespace b200 {

// Two E4M3 bytes (low 16 bits of s) -> bf16x2 (exact: E4M3 has 4 significant bits).
DEV uint32_t e4m3x2_to_bf16x2(uint32_t s) {
  uint32_t h;
  asm("{\n\t.reg .b16 t;\n\tcvt.u16.u32 t, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, t;\n\t}" : "=r"(h) : "r"(s & 0xFFFFu));
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&b);
}

// Four E2M1 codes (the four nibbles of the low 16 bits of w) -> two bf16x2 words, with byte permutes only: the
// conversion instructions (cvt e2m1x2 -> f16x2 -> f32 -> bf16x2, two per weight) run at a fraction of the ALU rate and
// were the bound of this kernel. The bf16 image of magnitude code c is {0, 0x3F00, 0x3F80, 0x3FC0, 0x4000, 0x4040,
// 0x4080, 0x40C0}[c]: its low and high bytes are looked up with prmt in two 8-byte tables, the sign bits are moved to
// bit 7 of the high bytes with prmt's sign-replication mode, and a last pair of prmt interleaves low and high bytes.
DEV void e2m1x4_to_bf16x2(uint32_t w, uint32_t& v01, uint32_t& v23) {
  const uint32_t sel = w & 0x7777u;
  const uint32_t lo = __byte_perm(0xC0800000u, 0xC0804000u, sel);        // low bytes of codes 0..3 | 4..7
  uint32_t hi = __byte_perm(0x3F3F3F00u, 0x40404040u, sel);              // high bytes
  const uint32_t u = w & 0x8888u;                                        // byte k of u: sign of nibble 2k+1 in bit 7, of 2k in bit 3
  const uint32_t sgn = __byte_perm(u, u << 4, 0x9D8Cu);                  // byte i = 0xFF if nibble i is negative (msb replication)
  hi |= sgn & 0x80808080u;
  v01 = __byte_perm(lo, hi, 0x5140u);
  v23 = __byte_perm(lo, hi, 0x7362u);
}

}  // namespace b200
