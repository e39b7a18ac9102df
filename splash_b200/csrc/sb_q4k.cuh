// Q4_K super-blocks as operands of warp-level MMA, shared by the projection kernel and the MoE experts' kernels: the weight is
// sc q, an exact integer in fp16 built as (1024 + q) sc - 1024 sc, and the block's d and dmin are applied to fp32 sums.
#pragma once
#include "sb_ptx.cuh"

namespace sb {

struct Q4Scales {
  uint32_t mlo, blo, mhi, bhi, mn0, mn1;
  float d, ndmin;
};
// The two sub-blocks (2t, 2t+1) a lane multiplies, from a super-block's 16-byte header
// {d, dmin, 12 packed 6-bit scale/min bytes}.
__device__ __forceinline__ Q4Scales q4_scales(const uint4 hdr, uint32_t t) {
  const uint32_t sh = (t & 1) * 16;
  const uint32_t a = hdr.y >> sh, b = hdr.z >> sh, c = hdr.w >> sh;
  const uint32_t sc_lo = a & 0x3f3fu, mn_lo = b & 0x3f3fu;
  const uint32_t sc_hi = (c & 0x0f0fu) | ((a >> 2) & 0x3030u), mn_hi = ((c >> 4) & 0x0f0fu) | ((b >> 2) & 0x3030u);
  const uint32_t sc = t < 2 ? sc_lo : sc_hi, mn = t < 2 ? mn_lo : mn_hi;
  const uint32_t k1024 = 0x64006400u;
  // {0x6400 | byte, 0x6400 | byte} - 1024 = the byte as two exact halves.
  const uint32_t s0 = hsub2_u32(__byte_perm(sc, 0x64646464u, 0x4040), k1024);
  const uint32_t s1 = hsub2_u32(__byte_perm(sc, 0x64646464u, 0x4141), k1024);
  Q4Scales r;
  r.mn0 = hsub2_u32(__byte_perm(mn, 0x64646464u, 0x4040), k1024);
  r.mn1 = hsub2_u32(__byte_perm(mn, 0x64646464u, 0x4141), k1024);
  r.mlo = s0;
  r.blo = hmul2_u32(s0, 0xE400E400u);  // * -1024
  r.mhi = hmul2_u32(s1, 0x2C002C00u);  // * 1/16
  r.bhi = hmul2_u32(s1, 0xD400D400u);  // * -64
  const __half2 dd = *reinterpret_cast<const __half2 *>(&hdr.x);
  r.d = __low2float(dd);
  r.ndmin = -__high2float(dd);
  return r;
}

}  // namespace sb
