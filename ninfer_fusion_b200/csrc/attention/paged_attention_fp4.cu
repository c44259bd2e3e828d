// Split-KV paged attention for decode / small-T verify over nvfp4 pages, head_dim 256, groups of up to eight query heads.
//
// The products, their groups of sixteen and the order of all sums are those of paged_attention_mma.cu, so that the bits are the
// same; what differs is how the operands come about:
//   * everything is transposed, S^T[16 keys, 8 heads] = K Q^T and O^T[16 d, 8 heads] += V^T P^T: the eight rows of a
//     16-row operand that stood empty there hold keys and columns, and half of the products go;
//   * K never sees shared memory.  A thread loads a quarter of its two keys' codes and trades bytes with its neighbour, after
//     which it holds what the operand's layout asks of it: of the sixteen dimensions of a product (halves of two neighbouring
//     16-value units; in which order they are summed makes no difference to a product) any four per thread.
// 8 sequences of up to 32,000 keys, 24 heads in 4 groups, 240 MB of cache (37 us): 145 us by the general kernel, bound by its
// issue slots (6000 a tile of 64 keys, 50 %) and shared memory (1550 wavefronts a tile, 58 %); now 105, 3500 and 800, and the
// latencies between two barriers with the sixteen warps that the registers admit.  Of these 40 us the conversion of a word of codes in one
// statement gave 10, K past shared memory 10, one barrier per tile for four and the transposed products 15, the second product by
// the V group alone, which waited for the other, 6.  32 sequences of 2600 keys 54 -> 42.
// Warps 0..3: K, S and softmax of sixteen keys of a tile each; 4..7: V as fp16 into shared memory, page look-ups, O of 64 columns
// each.  One barrier per tile: between two of them the probabilities of tile i, V of tile i, the scores of tile i + 1
// and the product of P and V of tile i - 1 are made.
#include "attention.h"

#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <math_constants.h>

#include "../common/ptx.cuh"
#include "../kv/codec.cuh"
#include "attn_mma_common.cuh"

namespace nfb {

namespace {

using namespace attn_mma;

constexpr int kThreads = 256;
constexpr int kGroup = kThreads / 2;             // threads of K (warps 0..3) and of V (warps 4..7)
constexpr int kRows = 8;                         // query heads, zero padded
constexpr int kWarpKeys = kTileKeys / 4;         // keys whose rows a warp converts
constexpr int kUnits = kTileKeys * 16 / kGroup;  // 16-value units of V per thread and tile

struct Smem {
  __half v[2][kTileKeys][kLdK];           // [tile mod 2], columns in the order of `dim_at`
  __half q[kRows][kLdQ];
  __half p[2][kRows][kLdP];               // [tile mod 2]
  float rowmax[2][4][kRows];              // [tile mod 2], per warp of the K group
  float rowsum[kTileKeys / 8][kRows];     // per eight keys of a tile
  alignas(16) int rows[4][kTileKeys];     // [tile mod 4]: cache rows (fewer than 2^31: they have 144 bytes), -1: none; see row_slot
  uint32_t all[4][2];                     // whether all keys of a half tile have rows
};
// place of a key's row in `rows`: a warp's even keys before its odd ones
__device__ __forceinline__ int row_slot(int key) { return (key & ~15) | ((key & 1) << 3) | ((key >> 1) & 7); }
// the dimension at column c of a V row: the units' first eight values in the first half of the row, their second eight in the second
__device__ __forceinline__ int dim_at(int c) { return ((c & (D / 2 - 1)) >> 3) * 16 + (c / (D / 2)) * 8 + (c & 7); }
// bytes H and H + 2 of a word: two pairs of e2m1 codes
template <int H>
__device__ __forceinline__ void pairs_at(uint32_t w, uint32_t& first, uint32_t& second) {
  if constexpr (H == 0)
    asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %2;\n\tcvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, c;\n\t}"
        : "=r"(first), "=r"(second) : "r"(w));
  else
    asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %2;\n\tcvt.rn.f16x2.e2m1x2 %0, b;\n\tcvt.rn.f16x2.e2m1x2 %1, d;\n\t}"
        : "=r"(first), "=r"(second) : "r"(w));
}

__global__ void __launch_bounds__(kThreads, 2) paged_attn_fp4_kernel(const PagedAttnParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);

  pdl_launch_next();
  pdl_wait_prior();
  const int t = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.n_q_heads / p.n_kv_heads;
  const int kv_len = p.q_kv_len[t];
  const int seq = p.q_seq[t];
  // a sliding window drops the keys before kv_len - window; the split then starts at the window's edge
  const int k_begin = max(split * p.split_keys, p.window > 0 ? kv_len - p.window : 0);
  const int k_end = min(kv_len, (split + 1) * p.split_keys);
  const long long part_base = (static_cast<long long>(t) * p.n_q_heads + kvh * G) * p.n_splits + split;

  if (seq < 0 || k_begin >= k_end) {
    for (int g = threadIdx.x; g < G; g += blockDim.x) {
      float* ml = p.part_ml + (part_base + static_cast<long long>(g) * p.n_splits) * 2;
      ml[0] = -CUDART_INF_F;
      ml[1] = 0.f;
    }
    return;
  }

  // Q rows (g < G valid, rest zero), pre-scaled so that softmax runs on exp2
  const float qscale = p.sm_scale * 1.4426950408889634f;
  for (int i = threadIdx.x; i < kRows * (D / 2); i += kThreads) {
    const int g = i / (D / 2), d2 = i % (D / 2);
    float2 f = make_float2(0.f, 0.f);
    if (g < G) {
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(
          p.q + (static_cast<long long>(t) * p.n_q_heads + kvh * G + g) * D + 2 * d2);
      f = make_float2(__bfloat162float(v.x) * qscale, __bfloat162float(v.y) * qscale);
    }
    *reinterpret_cast<uint32_t*>(&sm.q[g][2 * d2]) = pack_half2(f.x, f.y);
  }

  const unsigned long long tmask = p.tree_mask ? p.tree_mask[t] : ~0ull;
  const int tbase = p.tree_mask ? p.tree_base[t] : 0x7fffffff;
  const int* table = p.block_table + static_cast<long long>(seq) * p.table_stride;
  const int P = p.kv.page_size;
  const int n_tiles = (k_end - k_begin + kTileKeys - 1) / kTileKeys;
  const int row0 = lane >> 2, cq = lane & 3;   // accumulators: keys (or columns) row0 and row0 + 8, heads 2 cq and 2 cq + 1
  const bool is_v = warp >= 4;
  const int kw = warp & 3;

  // ---- rows: thread g < 64 of the V group finds key g of the tiles.  The page is asked for one tile before its row is published,
  //      the row three tiles ahead of its use.
  const int gtid = threadIdx.x & (kGroup - 1);
  int ask_key = k_begin + (gtid & (kTileKeys - 1)), ask_page = ask_key / P, ask_at = ask_key - ask_page * P, at = ask_at;
  int page_next = -1;
  auto next_page = [&] {
    page_next = gtid < kTileKeys && ask_key < k_end ? table[ask_page] : -1;   // (a released or unpublished page is -1 as well)
    ask_key += kTileKeys;
    at = ask_at;
    for (ask_at += kTileKeys; ask_at >= P; ask_at -= P) ++ask_page;
  };
  auto publish_row = [&](int i) {
    if (gtid < kTileKeys) {
      const int r = static_cast<int>(kv_row_of(p.kv, page_next, kvh, at));
      sm.rows[i & 3][row_slot(gtid)] = r;
      const bool all = __all_sync(0xffffffffu, r >= 0);
      if (lane == 0) sm.all[i & 3][gtid >> 5] = all;
    }
  };
  if (is_v) {
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
      next_page();
      publish_row(i);
    }
    next_page();
  }
  __syncthreads();

  float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.f, 0.f};
  float o[4][4];   // V group
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[m][j] = 0.f;

  const uint32_t p_addr = smem_u32(&sm.p[0][lane & 7][8 * (lane >> 3)]);
  const uint32_t v_addr = smem_u32(&sm.v[0][(lane & 7) + 8 * (lane >> 4)][kw * 64 + 8 * ((lane >> 3) & 1)]);
  // O^T[64 * kw .. + 63, :] += V^T P^T of tile i
  auto values = [&](int i) {
    const uint32_t v_tile = v_addr + (i & 1) * static_cast<int>(sizeof(sm.v[0]));
    const uint32_t p_tile = p_addr + (i & 1) * static_cast<int>(sizeof(sm.p[0]));
    uint32_t b[kTileKeys / 8];
#pragma unroll
    for (int k2 = 0; k2 < kTileKeys / 32; ++k2) ldmatrix_x4(p_tile + k2 * 64, b[4 * k2], b[4 * k2 + 1], b[4 * k2 + 2], b[4 * k2 + 3]);
#pragma unroll
    for (int kk = 0; kk < kTileKeys / 16; ++kk)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        uint32_t a[4];   // (V[key][d] is the transpose of the first operand)
        ldmatrix_x4_trans(v_tile + kk * 16 * kLdK * 2 + m * 32, a[0], a[1], a[2], a[3]);
        mma_f16(o[m], a[0], a[1], a[2], a[3], b[2 * kk], b[2 * kk + 1]);
      }
  };
  // the maxima of tile i: O and (`fade`, for the thread's row) the sums are faded where one has grown
  auto raise = [&](int i) {
    float fade = 1.f, corr[2];
    bool moved = false;
    float2 mt = *reinterpret_cast<const float2*>(&sm.rowmax[i & 1][0][2 * cq]);
#pragma unroll
    for (int w = 1; w < 4; ++w) {
      const float2 m = *reinterpret_cast<const float2*>(&sm.rowmax[i & 1][w][2 * cq]);
      mt.x = fmaxf(mt.x, m.x);
      mt.y = fmaxf(mt.y, m.y);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float mn = fmaxf(m_run[e], e ? mt.y : mt.x);
      moved |= mn != m_run[e];
      corr[e] = m_run[e];
      m_run[e] = mn;
    }
    if (__any_sync(0xffffffffu, moved)) {   // (where no maximum has grown the factors are ones)
#pragma unroll
      for (int e = 0; e < 2; ++e) corr[e] = m_run[e] == -CUDART_INF_F ? 1.f : exp2f(corr[e] - m_run[e]);
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[m][j] *= corr[j & 1];
      fade = row0 & 1 ? corr[1] : corr[0];
    }
    return fade;
  };

  if (is_v) {
    // =========================== V: sixteen values of every second of the warp's keys ===========================
    const int part = lane & 15;
    uint2 code[kUnits];
    uint32_t scale[kUnits];
    const uint8_t* const codes = p.kv.v_codes + part * 8;
    const uint8_t* const scales = p.kv.v_scales + part;
    auto load = [&](int i) {
      const int4* r4 = reinterpret_cast<const int4*>(&sm.rows[i & 3][kw * kWarpKeys + (lane >> 4) * 8]);
      const int4 ra = r4[0], rb = r4[1];
      const int r[kUnits] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
#pragma unroll
      for (int j = 0; j < kUnits; ++j) {
        code[j] = *reinterpret_cast<const uint2*>(codes + static_cast<long long>(max(r[j], 0)) * (D / 2));
        scale[j] = scales[static_cast<long long>(max(r[j], 0)) * (D / 16)];
      }
    };
    load(0);
    __half* const place = &sm.v[0][kw * kWarpKeys + (lane >> 4)][part * 8];
    __syncthreads();
#pragma unroll 1
    for (int i = 0; i < n_tiles; ++i) {
      // Since the last barrier everybody sees the maxima of tile i, and V and P of tile i - 1.
      if (i > 0) values(i - 1);
      raise(i);
      if (!(sm.all[i & 3][0] & sm.all[i & 3][1])) {
#pragma unroll 1
        for (int j = 0; j < kUnits; ++j)
          if (sm.rows[i & 3][kw * kWarpKeys + (lane >> 4) * 8 + j] < 0) {
#pragma unroll
            for (int k = 0; k < kUnits; ++k)
              if (k == j) code[k] = make_uint2(0, 0), scale[k] = 0;
          }
      }
#pragma unroll
      for (int j = 0; j < kUnits; ++j) {
        const __half2 s = e4m3_twice(scale[j]);
        uint4* dst = reinterpret_cast<uint4*>(place + (i & 1) * (kTileKeys * kLdK) + 2 * j * kLdK);
        const uint32_t w[2] = {code[j].x, code[j].y};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[4];
          e2m1_pairs(w[h], v);
          dst[h * (D / 16)] = make_uint4(mul_h2(v[0], s), mul_h2(v[1], s), mul_h2(v[2], s), mul_h2(v[3], s));
        }
      }
      if (i + 1 < n_tiles) load(i + 1);
      publish_row(i + 3);
      next_page();
      __syncthreads();
    }
  } else {
    // =========================== K, scores and softmax of the warp's sixteen keys ===========================
    // Thread cq of a key's four loads unit 4 j + 2 (cq & 1) + cq / 2, j = 0..3, and needs of all units 2 s + cq / 2, s = 0..7, the
    // bytes cq & 1 and 2 more of both halves: half of its own units' and half of its neighbour's.
    const int odd = cq & 1;
    uint32_t q[D / 8];   // Q of head row0, the four dimensions of each product
#pragma unroll
    for (int k = 0; k < D / 16; ++k) {
      const int d = (2 * (k & 7) + (cq >> 1)) * 16 + (k >> 3) * 8 + 2 * odd;
      q[2 * k] = *reinterpret_cast<const uint32_t*>(&sm.q[row0][d]);
      q[2 * k + 1] = *reinterpret_cast<const uint32_t*>(&sm.q[row0][d + 4]);
    }
    uint2 code[2][4];
    uint4 scale[2];
    const uint8_t* const codes = p.kv.k_codes + (2 * odd + (cq >> 1)) * 8;
    const uint8_t* const scales = p.kv.k_scales;
    auto load = [&](int i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long r = max(sm.rows[i & 3][row_slot(kw * kWarpKeys + row0 + 8 * h)], 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) code[h][j] = *reinterpret_cast<const uint2*>(codes + r * (D / 2) + j * 32);
        scale[h] = *reinterpret_cast<const uint4*>(scales + r * (D / 16));
      }
    };
    const uint32_t keep = odd ? 0x7351 : 0x6240, give = odd ? 0x6240 : 0x7351;   // bytes (y, y + 4, y + 2, y + 6) of the halves' words
    const uint32_t pick = 0x4440 + (cq >> 1);                                    // scale bytes of even units, or of odd ones
    float s[4];
    auto scores = [&](int i) {
      if (!(sm.all[i & 3][0] & sm.all[i & 3][1])) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (sm.rows[i & 3][row_slot(kw * kWarpKeys + row0 + 8 * h)] >= 0) continue;
#pragma unroll
          for (int j = 0; j < 4; ++j) code[h][j] = make_uint2(0, 0);
          scale[h] = make_uint4(0, 0, 0, 0);
        }
      }
      uint32_t w[2][8];
      __half2 sc[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t mine = __byte_perm(code[h][j].x, code[h][j].y, keep);
          const uint32_t other = __shfl_xor_sync(0xffffffffu, __byte_perm(code[h][j].x, code[h][j].y, give), 1);
          w[h][2 * j] = odd ? other : mine;
          w[h][2 * j + 1] = odd ? mine : other;
        }
        const uint32_t sw[4] = {scale[h].x, scale[h].y, scale[h].z, scale[h].w};
#pragma unroll
        for (int u = 0; u < 8; ++u) sc[h][u] = e4m3_twice(__byte_perm(sw[u >> 1], 0, pick + (u & 1) * 2));
      }
      if (i + 1 < n_tiles) load(i + 1);
      float s2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) s[j] = s2[j] = 0.f;
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        const int u = k & 7;
        uint32_t a[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (k < 8) pairs_at<0>(w[h][u], a[h], a[2 + h]);
          else pairs_at<1>(w[h][u], a[h], a[2 + h]);
          a[h] = mul_h2(a[h], sc[h][u]);
          a[2 + h] = mul_h2(a[2 + h], sc[h][u]);
        }
        mma_f16(k & 1 ? s2 : s, a[0], a[1], a[2], a[3], q[2 * k], q[2 * k + 1]);
      }
      float mx[2];
#pragma unroll
      for (int j = 0; j < 4; ++j) s[j] = s[j] + s2[j];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int key = k_begin + i * kTileKeys + kw * kWarpKeys + row0 + 8 * h;
        bool seen = key < k_end;
        if (seen && key >= tbase) seen = (tmask >> (key - tbase)) & 1ull;
        if (!seen) s[2 * h] = s[2 * h + 1] = -CUDART_INF_F;
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        mx[e] = fmaxf(s[e], s[2 + e]);
#pragma unroll
        for (int x = 4; x < 32; x *= 2) mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], x));
      }
      if (lane < 4) *reinterpret_cast<float2*>(&sm.rowmax[i & 1][kw][2 * cq]) = make_float2(mx[0], mx[1]);
    };
    load(0);
    scores(0);
    __syncthreads();
#pragma unroll 1
    for (int i = 0; i < n_tiles; ++i) {
      const float fade = raise(i);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float e[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) e[j] = s[2 * h + j] == -CUDART_INF_F ? 0.f : exp2f(s[2 * h + j] - m_run[j]);
        // sums go by pairs of neighbouring keys: the even key's thread adds up row 2 cq, the odd one's row 2 cq + 1
        const float other = __shfl_xor_sync(0xffffffffu, row0 & 1 ? e[0] : e[1], 4);
        l_run[h] = fmaf(l_run[h], fade, row0 & 1 ? other : e[0]);
        l_run[h] += row0 & 1 ? e[1] : other;
#pragma unroll
        for (int j = 0; j < 2; ++j) sm.p[i & 1][2 * cq + j][kw * kWarpKeys + row0 + 8 * h] = __float2half_rn(e[j]);
      }
      if (i + 1 < n_tiles) scores(i + 1);
      __syncthreads();
    }
    // row sums: over the key pairs of eight keys
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float l = l_run[h];
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      if (lane < 8) sm.rowsum[2 * kw + h][2 * cq + (row0 & 1)] = l;
    }
  }
  __syncthreads();
  if (!is_v) return;
  values(n_tiles - 1);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int g = 2 * cq + e;
    if (g >= G) continue;
    const long long pb = part_base + static_cast<long long>(g) * p.n_splits;
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) p.part_o[pb * D + dim_at(kw * 64 + m * 16 + 8 * h + row0)] = o[m][2 * h + e];
    if (kw == 0 && row0 == 0) {
      p.part_ml[pb * 2] = m_run[e];
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < kTileKeys / 8; ++w) tot += sm.rowsum[w][g];
      p.part_ml[pb * 2 + 1] = tot;
    }
  }
}

}  // namespace

// Returns cudaErrorNotSupported when the problem is outside this kernel (the caller takes the one of paged_attention_mma.cu).
cudaError_t paged_attention_fp4_split(const PagedAttnParams& p, cudaStream_t stream, bool pdl) {
  const int G = p.n_q_heads / p.n_kv_heads;
  // A thread reads the sixteen scales of a row at once.  From splits of four tiles on: with one or two its start and end cost more than
  // it gives (us, general kernel and this one: 6 heads over 1, splits of 128 keys, one sequence of 64 keys 6.0 and 6.5, 32 of 500 8.5 and
  // 9.7, 32 of 1500 16.0 and 16.7; 24 over 4, one of 2048 9.1 and 9.3; splits of 256, one of 20000 30.7 -> 27.8, 8 of 4000 27.8 -> 24.6).
  if (p.split_keys < 4 * kTileKeys || p.kv.format != kKvNvfp4 || p.head_dim != D || G > kRows || p.split_keys % kTileKeys ||
      reinterpret_cast<uintptr_t>(p.kv.k_scales) % 16)
    return cudaErrorNotSupported;
  static const cudaError_t attr =
      cudaFuncSetAttribute(paged_attn_fp4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(Smem)));
  if (attr != cudaSuccess) return attr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.Tq, p.n_kv_heads, p.n_splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(Smem);
  cfg.stream = stream;
  cudaLaunchAttribute launch_attr[1];
  launch_attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  launch_attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = launch_attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, paged_attn_fp4_kernel, p);
}

}  // namespace nfb
