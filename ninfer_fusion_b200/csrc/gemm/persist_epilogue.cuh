// Epilogue of the persistent GEMM kernels (eight warps, 2..9): their barriers, and the way of a chunk of sixteen tokens between a
// warp's registers and rows in memory.
//
// A lane holds one weight row n = output column and sixteen tokens; rows of the output run along n.  The two lanes of a pair (n,
// n + 1) swap halves of packed words, so that the even lane stores both columns of tokens 0, 2, .. and the odd one of tokens 1, 3,
// ..: eight 4-byte stores of 2 x 64 bytes a warp.  Pointers step by two rows and full chunks have no predicates.  A token's row
// offset as a product and two comparisons per store made 375 instructions a chunk, and a tile of 128 x 256 took 6.4 us (bf16 store,
// one k-block of 64 with it), as long as the main loop of K = 1100; so it is 3.5.
#pragma once
#include <stdint.h>

#include <cuda_bf16.h>

namespace nfb {

// AND of a predicate over the epilogue warps (and a barrier of them)
__device__ __forceinline__ bool epi_all(bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, 1, 256, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(r) : "r"(static_cast<uint32_t>(v)) : "memory");
  return r != 0;
}
// the two warps of pair 0..3 (gate rows and the matching up rows of the same token columns)
__device__ __forceinline__ void epi_pair_sync(int pair) { asm volatile("bar.sync %0, 64;" ::"r"(2 + pair) : "memory"); }

// (a token pair of this lane's column) <-> (a column pair of this lane's token), see above
__device__ __forceinline__ uint32_t swap_pair(uint32_t w, uint32_t select) {
  return __byte_perm(w, __shfl_xor_sync(0xffffffffu, w, 1), select);
}
__device__ __forceinline__ uint32_t swap_select(int lane) { return (lane & 1) ? 0x3276u : 0x5410u; }

// Rows of a chunk as one lane reads and writes them: `at` = address of its first token's column pair (token lane & 1 of the
// chunk), `step` = two rows, in elements; `live` = how many of its up to eight rows exist.
struct ChunkRows {
  const __nv_bfloat16* at;
  long long step;
  int live;
};
__device__ __forceinline__ void load_rows8(const ChunkRows& r, uint32_t* w) {
  const __nv_bfloat16* at = r.at;
  if (r.live >= 8) {
#pragma unroll
    for (int m = 0; m < 8; ++m, at += r.step) w[m] = *reinterpret_cast<const uint32_t*>(at);
  } else {
#pragma unroll
    for (int m = 0; m < 8; ++m, at += r.step) w[m] = m < r.live ? *reinterpret_cast<const uint32_t*>(at) : 0u;
  }
}
// N = 4: a chunk of eight tokens
template <int N = 8>
__device__ __forceinline__ void store_rows(const ChunkRows& r, const uint32_t* w) {
  __nv_bfloat16* at = const_cast<__nv_bfloat16*>(r.at);
  if (r.live >= N) {
#pragma unroll
    for (int m = 0; m < N; ++m, at += r.step) *reinterpret_cast<uint32_t*>(at) = w[m];
  } else {
#pragma unroll
    for (int m = 0; m < N; ++m, at += r.step)
      if (m < r.live) *reinterpret_cast<uint32_t*>(at) = w[m];
  }
}
// sixteen tokens of this lane's column, plus the residual's words if there are any, rounded and stored
template <bool RESID>
__device__ __forceinline__ void store_chunk(const ChunkRows& r, const float* f, const uint32_t* resid, uint32_t select) {
  uint32_t w[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    float a = f[2 * m], b = f[2 * m + 1];
    if constexpr (RESID) {
      const uint32_t x = swap_pair(resid[m], select);
      a += __uint_as_float(x << 16);
      b += __uint_as_float(x & 0xffff0000u);
    }
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    w[m] = swap_pair(*reinterpret_cast<const uint32_t*>(&v), select);
  }
  store_rows(r, w);
}

}  // namespace nfb
