// One 16-value block of an nvfp4 (W4A4) activation row: e4m3 block scale = amax / 6, e2m1 codes, and the place of both
// in the operand the block-scaled GEMM reads -- codes row-major [T][K / 2], scales in the 512-byte tiles of the
// scale plane (128 rows x 4 scales, the layout tcgen05.cp expects).  Shared by the stand-alone quantiser and by the
// producers that quantise their own output (SwiGLU epilogue, GDN step, attention merge), so that all of them write the
// same bits.
#pragma once
#include <stdint.h>

#include "../kv/codec.cuh"

namespace nfb {

constexpr int kNvfp4SfTileBytes = 512;   // 128 rows x 4 scales

// e2m1 code of v / s, to nearest, ties to even, for a bf16 v and an e4m3 s > 0.  The boundaries lie midway between the grid's
// values and have three significant bits at most, s has four, so that a boundary times s is exact and has seven; v has eight.  Two
// different numbers of eight bits lie at least 2^-8 of the larger apart, far more than the rounding of a quotient to fp32: comparing
// products gives what comparing that quotient gives, at a third of the instructions (quantiser, 2048 x 17408: 55 -> 33 us; 256 x 5120:
// 6.9 -> 4.6).
__device__ __forceinline__ uint32_t e2m1_code(float v, float s) {
  const float a = fabsf(v);
  // (as negations: a NaN takes the largest code)
  const uint32_t m = !(a <= 0.25f * s) + !(a < 0.75f * s) + !(a <= 1.25f * s) + !(a < 1.75f * s) + !(a <= 2.5f * s) +
                     !(a < 3.5f * s) + !(a <= 5.f * s);
  return m | (v < 0.f ? 8u : 0u);
}

// `v`: the block's sixteen values as the consumer would read them from a bf16 tensor (already rounded to bf16);
// token row t, block g of the row (K / 16 blocks per row).
__device__ __forceinline__ void nvfp4_store_block(const float* v, int t, int g, int K, uint8_t* codes, uint8_t* sf_plane) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  const uint8_t sc = float_to_e4m3(amax / 6.f);
  const float sf = e4m3_to_float(sc);
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    lo |= e2m1_code(v[i], sf) << (4 * i);
    hi |= e2m1_code(v[8 + i], sf) << (4 * i);
  }
  if (!(sf > 0.f)) lo = hi = 0;
  *reinterpret_cast<uint2*>(codes + static_cast<long long>(t) * (K / 2) + g * 8) = make_uint2(lo, hi);
  const int k_tiles = K / 64;
  const long long off = (static_cast<long long>(t / 128) * k_tiles + g / 4) * kNvfp4SfTileBytes + (t % 32) * 16 +
                        ((t % 128) / 32) * 4 + (g % 4);
  sf_plane[off] = sc;
}

}  // namespace nfb
