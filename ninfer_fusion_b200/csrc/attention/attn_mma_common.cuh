// Shared pieces of the tensor-core attention kernels over pages: tile geometry and ldmatrix / mma wrappers of the split-KV
// decode kernel, and the raw-unit loader that dequantises 16 cache values to fp16 pairs, which the prefill kernel takes too.
#pragma once
#include <cuda_fp16.h>
#include <cuda_fp4.h>
#include <stdint.h>

#include "../common/ptx.cuh"
#include "../kv/codec.cuh"

namespace nfb {
namespace attn_mma {

constexpr int D = 256;
constexpr int kTileKeys = 64;
constexpr int kLdK = D + 8;          // halves per K-tile row
constexpr int kLdP = kTileKeys + 8;
constexpr int kLdQ = D + 8;


__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// Codes to fp16 pairs, all of a word in one statement: bytes taken from it one by one, as the conversion functions take them, are
// shifted and masked before each conversion (a word of e2m1 codes and its four products 21 cycles of a scheduler, so 11).
__device__ __forceinline__ void e2m1_pairs(uint32_t w, uint32_t* out) {
  asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\tcvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
      : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3]) : "r"(w));
}
__device__ __forceinline__ void e4m3_pairs(uint32_t w, uint32_t* out) {
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, a;\n\tcvt.rn.f16x2.e4m3x2 %1, b;\n\t}"
      : "=r"(out[0]), "=r"(out[1]) : "r"(w));
}
// an e4m3 scale, twice
__device__ __forceinline__ __half2 e4m3_twice(uint32_t code) {
  const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(code * 0x101u), __NV_E4M3);
  return *reinterpret_cast<const __half2*>(&r);
}
__device__ __forceinline__ uint32_t mul_h2(uint32_t a, __half2 b) {
  const __half2 r = __hmul2(*reinterpret_cast<const __half2*>(&a), b);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// One "unit" = 16 consecutive values [16*part, 16*part+16) of a cache row.  Loading (raw bytes into
// registers) and converting (to 8 packed fp16 pairs) are separate so that a thread can put all of a
// tile's loads in flight before it converts the first one.  For that the loads are unconditional and nothing is done with
// their results before `convert`: a load under a condition, or a scale decoded where it is loaded, makes the thread wait
// for each unit in turn (128-key tiles of the prefill kernel: 3500 ns per tile so, 1700 without the wait).  A row that does
// not exist (r < 0) is read as row 0 and `clear`ed before it is converted.  The fp8-row scale is NOT applied here (it
// multiplies scores / probabilities instead).
template <int FORMAT>
struct RawUnit {
  uint4 a;
  uint4 b;         // second half of a bf16 unit only
  uint32_t scale;  // int8-group (fp16 bits) / nvfp4 (e4m3 code) block scale
  int tier;        // mixed layers: the tier this unit was read from (decides how it is converted)

  // `which` 0 = K, 1 = V; `r` as returned by kv_row_of (mixed layers: tier in the top bits)
  __device__ __forceinline__ void load_row(const KvLayer& kv, int which, long long r, int part) {
    r = r < 0 ? 0 : r;
    if constexpr (FORMAT == kKvMixed) {
      tier = kv_row_tier(r);
      const long long rr = kv_row_index(r);
      const uint8_t* codes = which ? kv.tier_v_codes[tier] : kv.tier_k_codes[tier];
      if (tier == 0) {
        const uint4* src = reinterpret_cast<const uint4*>(codes + rr * (2 * D) + part * 32);
        a = src[0];
        b = src[1];
      } else if (tier == 1) {
        a = *reinterpret_cast<const uint4*>(codes + rr * D + part * 16);
      } else {
        const uint2 c = *reinterpret_cast<const uint2*>(codes + rr * (D / 2) + part * 8);
        a = make_uint4(c.x, c.y, 0, 0);
        const uint8_t* scales = which ? kv.tier_v_scales[2] : kv.tier_k_scales[2];
        scale = scales[rr * (D / 16) + part];
      }
    } else {
      load(kv, which ? kv.v_codes : kv.k_codes, which ? kv.v_scales : kv.k_scales, r, part);
    }
  }
  __device__ __forceinline__ void load(const KvLayer& kv, const uint8_t* codes, const uint8_t* scales, long long r,
                                       int part) {
    if constexpr (FORMAT == kKvFp8Row) {
      a = *reinterpret_cast<const uint4*>(codes + r * D + part * 16);
    } else if constexpr (FORMAT == kKvBf16) {
      const uint4* src = reinterpret_cast<const uint4*>(codes + r * (2 * D) + part * 32);
      a = src[0];
      b = src[1];
    } else if constexpr (FORMAT == kKvInt8Group) {
      a = *reinterpret_cast<const uint4*>(codes + r * D + part * 16);
      scale = reinterpret_cast<const uint16_t*>(scales + r * (2 * (D / kv.group)))[part * 16 / kv.group];
    } else {
      const uint2 c = *reinterpret_cast<const uint2*>(codes + r * (D / 2) + part * 8);
      a.x = c.x;
      a.y = c.y;
      scale = scales[r * (D / 16) + part];
    }
  }
  // the unit of a row that does not exist: codes and a scale whose values are zeros
  __device__ __forceinline__ void clear() {
    a = b = make_uint4(0, 0, 0, 0);
    scale = 0;
  }
  __device__ __forceinline__ void convert(uint32_t* out) const {
    if constexpr (FORMAT == kKvMixed) {
      // one of the three tier codecs, chosen per unit
      if (tier == 0) {
        RawUnit<kKvBf16> u;
        u.a = a; u.b = b;
        u.convert(out);
      } else if (tier == 1) {
        RawUnit<kKvFp8Row> u;
        u.a = a;
        u.convert(out);
      } else {
        RawUnit<kKvNvfp4> u;
        u.a = a; u.scale = scale;
        u.convert(out);
      }
    } else if constexpr (FORMAT == kKvFp8Row) {
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) e4m3_pairs(w[i], out + 2 * i);
    } else if constexpr (FORMAT == kKvBf16) {
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
        out[i] = pack_half2(__bfloat162float(v.x), __bfloat162float(v.y));
      }
    } else if constexpr (FORMAT == kKvInt8Group) {
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
      const __half2 s2 = __half2half2(__ushort_as_half(static_cast<unsigned short>(scale)));
      // A code plus 128 under the exponent of 1024 is the fp16 number 1152 + code: two bytes become a pair with one byte
      // permutation and a subtraction that is exact.  The product with the fp16 scale is rounded once, as through fp32.
      const __half2 bias = __half2half2(__ushort_as_half(0x6480));
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t b = __byte_perm(w[i / 2] ^ 0x80808080u, 0x64646464u, i % 2 ? 0x4342 : 0x4140);
        const __half2 h = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&b), bias), s2);
        out[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
    } else {
      // two e2m1 codes per byte -> fp16 pair in one conversion instruction, then the block scale (the product of an
      // e2m1 value and an e4m3 scale is exact in fp16, so this equals the fp32 route bit for bit)
      const __half2 s2 = e4m3_twice(scale);
      e2m1_pairs(a.x, out);
      e2m1_pairs(a.y, out + 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = mul_h2(out[i], s2);
    }
  }
};

}  // namespace attn_mma
}  // namespace nfb
