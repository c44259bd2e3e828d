// Causal paged attention for prefill chunks and wide verify passes (head_dim 256) on the 5th-generation tensor cores.
//
// One CTA = one block of consecutive query tokens of one sequence x one KV head.  The 128 MMA rows are (query token,
// query head of the GQA group) pairs; keys come in tiles of 64:
//
//   S[128 rows, 64 keys] = Q . K^T     Q in TMEM (fp16), K in shared memory (fp16, K-major, 128-byte swizzle), S in TMEM
//   O[128 rows, 256 d]  += P . V       P in TMEM (fp16, over the S it came from), V in shared memory as it lies in the
//                                      page ([key][d] = an MN-major operand: no transpose), O in TMEM
//
// Seventeen warps:
//   0..7    softmax, two threads per row: Q into TMEM, then per tile the row maximum, exp2, P back to TMEM, the row sum in
//           registers; at the end the normalised row.  Of every eight keys one thread takes the first four and the other the rest
//   8..11   K: rows of a tile gathered from their pages into registers up to two tiles ahead of their use, dequantised once
//           (bf16 / fp8-row / int8-group / nvfp4 -> fp16) into one of two shared-memory slots
//   12..15  V, the same way; 8..15 also load the output gate beside the last products and store the result
//   16      issues the products: S of tile i + 1 goes in front of P V of tile i, so that the softmax of one tile runs beside
//           the products of its neighbours
// The row scales of fp8 pages never touch the operands: the K scale multiplies a key's column of S, the V scale its
// probability.  A row's exponentials are taken against its largest score so far, so that no probability exceeds one (times an
// fp8 V scale: at most 65504, fp16's largest; below, values of a page row that are all under 0.027 have scales under 2^-14, whose
// products fp16 holds with fewer bits, and drops below 2^-25); O is rescaled in TMEM by the warps that have a row whose maximum
// has grown.  K / V of the chunk itself were appended by attn_prep before this kernel runs, so the key loop covers [first
// visible key, last visible key] with a limit per row.
//
// TMEM is full (two S buffers of 64 columns, Q 128, O 256).  Q lies there and not in shared memory because the gathers need
// the room: with Q and 128-key K and V tiles in shared memory (192 KB) 28 KB of L1 were left, which bound the loads in flight
// and with them the kernel (4.2 us per 128 keys; the products alone take 1.6).  Then the serial chain scores -> softmax -> P of
// a tile bounds it, with one thread per row, and instructions: of the four schedulers one had the issuer, a softmax, a K and a V
// warp to choose from, and divisions by the page size, selects per row and stores with two-way conflicts to issue (issue slots
// 54 %, the integer units 45 %, a fifth of the stalls for instructions not yet fetched).  Two threads per row, pages walked
// without a division, row numbers of 32 bits, the check for keys without a row once per tile and conflict-free stores: 24 / 4
// heads, 2048 queries, us, before -> now: 2048 keys, fp8 rows 161 -> 123, bf16 164 -> 131, nvfp4 152 -> 110, int8 174 -> 141;
// 16384 keys, fp8 rows 1367 -> 1097 (705 TFLOP/s), bf16 1526 -> 1265, nvfp4 1337 -> 952, int8 1696 -> 1454; 300 queries, 1500
// keys 68 -> 55; 37 tokens, of which a launch is the most, 21.5 -> 15.7; bits are the same.  Left: 3.3 us per 128 keys, the
// chain of a tile still (a maximum that lags by up to four powers of two would spare a tenth of it, with other roundings).
//
// Reference kernels covered: kernel/gqa_attention_prefill_{bf16,i8,nvfp4}.cuh (Br = 64 x Bc = 64
// mma.sync kernels that also quantise-append in-kernel).
#include "attention.h"

#include <math_constants.h>

#include <type_traits>

#include "../common/quotient.cuh"
#include "attn_mma_common.cuh"

namespace nfb {

namespace {

using attn_mma::D;
using attn_mma::RawUnit;
using attn_mma::pack_half2;

constexpr int kRows = 128;                   // MMA rows: (query token, head) pairs
constexpr int kKeys = 64;                    // keys per tile
constexpr int kAtomBytes = kKeys * 128;      // 64 columns of d: [64 keys][128 bytes], 8-row swizzle atoms of 1024 bytes
constexpr int kTileBytes = 4 * kAtomBytes;   // one [64][256] fp16 operand
constexpr int kSmemBytes = 4 * kTileBytes + 1024;   // two slots of K, two of V
constexpr int kGroup = 128;                  // threads of the K and V groups, and of each half of the softmax
constexpr int kSoftmax = 2 * kGroup;
constexpr int kThreads = kSoftmax + 2 * kGroup + 32;
constexpr int kIssuer = kThreads / 32 - 1;   // warp that issues the products
constexpr int kHalfKeys = kKeys / 2;
constexpr int kUnits = kKeys * 16 / kGroup;  // 16-value units per thread and tile
constexpr int kStagePitch = 2 * D + 16;      // bytes per row of the output tile: neighbouring rows start in other banks
constexpr uint32_t kColQ = 128, kColO = 256; // TMEM: S / P of even tiles at 0, of odd tiles at 64, then Q and O
constexpr uint32_t kIdescS = umma_idesc(128, kKeys, 0, 0);
constexpr uint32_t kIdescPV = umma_idesc(128, D, 0, 0) | (1u << 16);   // B (= V) is MN-major
enum : int { kStatusPrefillWait = 6 };

struct Bars {
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_done;
};

__device__ __forceinline__ uint64_t desc_v(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(kAtomBytes >> 4) << 16;   // next 64 columns of d
  d |= static_cast<uint64_t>(1024 >> 4) << 32;         // next 8 keys
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// D[tmem] (+)= A[tmem] * B[smem], fp16 inputs: A holds two consecutive k per 32-bit column
__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
        "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
        "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait_x32(uint32_t* r) {
  tmem_ld_wait_x16(r);
  asm volatile("" : "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
               "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}
__device__ __forceinline__ void tmem_ld_x4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_x2(uint32_t taddr, uint32_t a, uint32_t b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two floats in one instruction
__device__ __forceinline__ void mul2(uint32_t& x, uint32_t& y, float a, float b) {
  asm("{\n\t.reg .b64 u, w;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 w, {%2, %3};\n\tmul.rn.f32x2 u, u, w;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "+r"(x), "+r"(y) : "f"(a), "f"(b));
}
__device__ __forceinline__ void add2(float& x, float& y, float a, float b) {
  asm("{\n\t.reg .b64 u, w;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 w, {%2, %3};\n\tadd.rn.f32x2 u, u, w;\n\tmov.b64 {%0, %1}, u;\n\t}"
      : "+f"(x), "+f"(y) : "f"(a), "f"(b));
}
__device__ __forceinline__ void group_bar(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
// 16 bytes of a bf16 row: rows at any even element address are accepted, 16-byte accesses are used where all of them are aligned
__device__ __forceinline__ uint4 load_row16(const __nv_bfloat16* src, bool wide) {
  if (wide) return *reinterpret_cast<const uint4*>(src);
  const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
  return make_uint4(s[0], s[1], s[2], s[3]);
}
__device__ __forceinline__ void store_row16(__nv_bfloat16* dst, uint4 v, bool wide) {
  if (wide) {
    *reinterpret_cast<uint4*>(dst) = v;
  } else {
    uint32_t* d = reinterpret_cast<uint32_t*>(dst);
    d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
  }
}

// The page of a key and its place there, for keys that come a tile apart (page sizes need not divide a tile or be divided by it).
struct PageWalk {
  int page, at;
  __device__ __forceinline__ PageWalk(int key, int size) : page(key / size), at(key - key / size * size) {}
  __device__ __forceinline__ void next_tile(int size) {
    at += kKeys;
    while (at >= size) {
      at -= size;
      ++page;
    }
  }
};

template <int FORMAT>
__global__ void __launch_bounds__(kThreads, 1) paged_attn_prefill_kernel(const PrefillAttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) Bars bars;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  // (rows have 144 bytes or more: 2^31 of them are more than the memory; a mixed layer's carry their tier in the top bits)
  using Row = std::conditional_t<FORMAT == kKvMixed, long long, int>;
  __shared__ Row rows_s[2][4][kKeys];                        // [K, V][tile mod 4]: cache rows of the tile's keys, -1: none
  __shared__ uint32_t all_s[2][4][2];                        // whether all keys of a half tile have rows
  __shared__ __align__(16) float scale_s[2][2][kKeys];       // [tile parity][K, V]
  __shared__ float half_s[2][2][kRows];                      // [tile parity][half]: what the halves of a row tell one another
  constexpr bool kScaled = FORMAT == kKvFp8Row || FORMAT == kKvMixed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abortp = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bars.k_full[b]), 4);
      mbar_init(smem_u32(&bars.k_empty[b]), 1);
      mbar_init(smem_u32(&bars.v_full[b]), 4);
      mbar_init(smem_u32(&bars.v_empty[b]), 1);
      mbar_init(smem_u32(&bars.s_full[b]), 1);
      mbar_init(smem_u32(&bars.p_full[b]), kSoftmax / 32);
    }
    mbar_init(smem_u32(&bars.o_done), 1);
    mbar_fence_init();
  }
  if (warp == kIssuer) {
    tmem_alloc(smem_u32(&tmem_base_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot;
  pdl_launch_next();
  pdl_wait_prior();

  // Longest first: a later query block of a causal prompt sees more keys, and CTAs are handed out in grid order, so
  // the grid runs the blocks from the last to the first (all KV heads of a block side by side); the short blocks
  // then fill the tail of the last wave instead of one long block running alone.
  const int kvh = blockIdx.x, blk = static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y);
  const int G = p.n_q_heads / p.n_kv_heads;
  const int t0 = p.blk_start[blk];
  const int n_tok = p.blk_count[blk];
  const int seq = n_tok > 0 ? p.q_seq[t0] : -1;
  const int n_rows = seq >= 0 ? n_tok * G : 0;
  const int k_end = n_rows > 0 ? p.q_kv_len[t0 + n_tok - 1] : 0;  // the last token of the block sees the most keys
  // sliding window: row r sees keys [lim - window, lim); tiles entirely before the first token's window are skipped
  const int k_first = n_rows > 0 && p.window > 0 ? max(0, p.q_kv_len[t0] - p.window) / kKeys * kKeys : 0;
  const int n_tiles = n_rows > 0 ? max(0, k_end - k_first + kKeys - 1) / kKeys : 0;
  const int* table = p.block_table + static_cast<long long>(max(seq, 0)) * p.table_stride;
  const int P = p.kv.page_size;
  const bool wide = ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.gate) |
                      static_cast<uintptr_t>(p.ld_gate * 2)) & 15) == 0;
  uint8_t* const stage = smem_gen;   // output tile, over the K and V slots once every product has retired

  if (warp == kIssuer) {
    // =========================== issuer of the products ===========================
    if (elect_one()) {
      auto scores = [&](int i) {
        const int b = i & 1;
        if (!mbar_wait(smem_u32(&bars.k_full[b]), (i >> 1) & 1, abortp, p.status, kStatusPrefillWait)) return false;
        tc_fence_after();
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint64_t kd = umma_desc_k_sw128(smem_base + b * kTileBytes + a * kAtomBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f16_ts(tmem + b * kKeys, tmem + kColQ + 8 * (4 * a + k), kd + 2 * k, kIdescS, (a | k) ? 1u : 0u);
        }
        tc_commit(smem_u32(&bars.s_full[b]));
        tc_commit(smem_u32(&bars.k_empty[b]));
        return true;
      };
      // Q is in TMEM: the softmax threads say so with the first arrivals on P's odd barrier
      bool ok = n_tiles > 0 && mbar_wait(smem_u32(&bars.p_full[1]), 0, abortp, p.status, kStatusPrefillWait) && scores(0);
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int b = i & 1;
        // The buffer of S(i + 1) holds P(i - 1) until that tile's product has read it: products with unlike accumulators and
        // shapes may pass one another.
        if (i > 0 && i + 1 < n_tiles &&
            !mbar_wait(smem_u32(&bars.v_empty[b ^ 1]), ((i - 1) >> 1) & 1, abortp, p.status, kStatusPrefillWait)) break;
        if (i + 1 < n_tiles && !scores(i + 1)) break;
        if (!mbar_wait(smem_u32(&bars.v_full[b]), (i >> 1) & 1, abortp, p.status, kStatusPrefillWait)) break;
        if (!mbar_wait(smem_u32(&bars.p_full[b]), ((i >> 1) + b) & 1, abortp, p.status, kStatusPrefillWait)) break;
        tc_fence_after();
        const uint64_t vd = desc_v(smem_base + (2 + b) * kTileBytes);
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k)
          mma_f16_ts(tmem + kColO, tmem + b * kKeys + 8 * k, vd + k * (2048 >> 4), kIdescPV, (i | k) ? 1u : 0u);
        tc_commit(smem_u32(&bars.v_empty[b]));
        // (a barrier of its own: when the softmax of the last tile is done, two products may be outstanding, and a parity
        // only tells neighbouring phases apart)
        if (i + 1 == n_tiles) tc_commit(smem_u32(&bars.o_done));
      }
    }
    __syncwarp();
  } else if (warp >= kSoftmax / 32) {
    // =========================== K (warps 8..11) and V (warps 12..15) ===========================
    // A wait that runs out sets the abort word and the status; the loop goes on, so that the group's barriers stay uniform.
    const int which = warp >= 12 ? 1 : 0, gtid = threadIdx.x & (kGroup - 1);
    // tiles in registers: the gathers of a tile are issued when the tile `kSets` before it has been converted (bf16 units are
    // 32 bytes each: one tile fits)
    constexpr int kSets = FORMAT == kKvBf16 || FORMAT == kKvMixed ? 1 : 2;
    RawUnit<FORMAT> raw[kSets][kUnits];
    uint32_t live[kSets];   // bit per unit: its row exists
    // page of this thread's key of the next tile asked for (-1: none, or released: its rows are zero), and the row behind it
    PageWalk ask(k_first + (gtid & (kKeys - 1)), P), place = ask;
    int ask_key = k_first + gtid;
    auto next_page = [&] {
      const int page = gtid < kKeys && ask_key < k_end ? table[ask.page] : -1;
      ask_key += kKeys;
      ask.next_tile(P);
      return page;
    };
    auto publish_row = [&](int i, int page) {
      if (gtid < kKeys) {
        const long long r = kv_row_of(p.kv, page, kvh, place.at);
        rows_s[which][i & 3][gtid] = static_cast<Row>(r);
        const bool all = __all_sync(0xffffffffu, r >= 0);
        if (lane == 0) all_s[which][i & 3][gtid >> 5] = all;
      }
      place.next_tile(P);
    };
    const uint8_t* const codes = which ? p.kv.v_codes : p.kv.k_codes;
    const uint8_t* const scales = which ? p.kv.v_scales : p.kv.k_scales;
    // Eight neighbouring lanes have four units of an even row and of the odd one behind it: the swizzle puts their halves into
    // eight bank groups.
    const int r0 = (gtid >> 5) * 2 + ((gtid >> 2) & 1), part = ((gtid >> 3) & 3) * 4 + (gtid & 3);
    const int chunk = (part & 3) * 2;
    uint8_t* const place0 = smem_gen + 2 * which * kTileBytes + (part >> 2) * kAtomBytes + r0 * 128;
    uint8_t* const lo0 = place0 + ((chunk ^ r0) << 4);
    uint8_t* const hi0 = place0 + (((chunk + 1) ^ r0) << 4);
    // unit j of a tile: this thread's sixteen columns of its key in the j-th eight
    auto load_unit = [&](int i, int j, RawUnit<FORMAT>& dst) {
      const Row r = rows_s[which][i & 3][8 * j + r0];
      if constexpr (FORMAT == kKvMixed) dst.load_row(p.kv, which, r, part);
      else dst.load(p.kv, codes, scales, max(r, 0), part);
    };
    auto store_unit = [&](const RawUnit<FORMAT>& src, int b, int j) {
      uint32_t h[8];
      src.convert(h);
      *reinterpret_cast<uint4*>(lo0 + b * kTileBytes + j * 1024) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(hi0 + b * kTileBytes + j * 1024) = make_uint4(h[4], h[5], h[6], h[7]);
    };
    auto live_units = [&](int i) {
      uint32_t m = (1u << kUnits) - 1;
      if (!(all_s[which][i & 3][0] & all_s[which][i & 3][1])) {
        m = 0;
#pragma unroll 1
        for (int j = 0; j < kUnits; ++j) m |= static_cast<uint32_t>(rows_s[which][i & 3][8 * j + r0] >= 0) << j;
      }
      return m;
    };
    int page_next = -1;
    if (n_tiles > 0) {
      int pages[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) pages[i] = next_page();
      page_next = next_page();
#pragma unroll
      for (int i = 0; i < 3; ++i) publish_row(i, pages[i]);
      group_bar(2 + which);
#pragma unroll
      for (int i = 0; i < kSets; ++i) {
        live[i] = live_units(i);
#pragma unroll
        for (int j = 0; j < kUnits; ++j) load_unit(i, j, raw[i][j]);
      }
    }
    auto step = [&](int i, RawUnit<FORMAT>* set, uint32_t& mask) {
      const int b = i & 1;
      const uint32_t freed = smem_u32(which ? &bars.v_empty[b] : &bars.k_empty[b]);
      if (i >= 2) mbar_wait(freed, ((i >> 1) - 1) & 1, abortp, p.status, kStatusPrefillWait);
      // With one set a unit's registers take the next tile as soon as it is converted (its rows were published long ago); with two
      // the loads wait for the last conversion, since one that waits for its data waits for the loads issued before it too
      // (2048 queries, 16384 keys: int8, interleaved, 3052 us where 1454; bf16, not, 1550 where 1265).
      uint32_t next_mask = 0;
      if (mask != (1u << kUnits) - 1) {
#pragma unroll
        for (int j = 0; j < kUnits; ++j)
          if (!(mask >> j & 1u)) set[j].clear();
      }
      if constexpr (kSets == 1) {
        const bool more = i + 1 < n_tiles;
        if (more) next_mask = live_units(i + 1);
#pragma unroll
        for (int j = 0; j < kUnits; ++j) {
          store_unit(set[j], b, j);
          if (more) load_unit(i + 1, j, set[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < kUnits; ++j) store_unit(set[j], b, j);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(which ? &bars.v_full[b] : &bars.k_full[b]));
      // rows of tile i + 3 from the page asked for a tile ago
      publish_row(i + 3, page_next);
      page_next = next_page();
      group_bar(2 + which);
      if constexpr (kSets == 1) {
        mask = next_mask;
      } else if (i + 2 < n_tiles) {
#pragma unroll
        for (int j = 0; j < kUnits; ++j) load_unit(i + 2, j, set[j]);
        mask = live_units(i + 2);
      }
    };
    for (int i = 0; i < n_tiles; i += kSets) {
      step(i, raw[0], live[0]);
      if constexpr (kSets == 2)
        if (i + 1 < n_tiles) step(i + 1, raw[1], live[1]);
    }
    // ---- the normalised rows from the stage, times the gate: four 16-byte pieces of a thread at a time, the first four gates
    //      loaded beside the last products.  (All sixteen in a row are code that every launch fetches anew: a prompt of 37 tokens,
    //      one key tile, took 59 us a layer so, 39 in a loop.) ----
    constexpr int kOut = kRows * (D / 8) / (2 * kGroup), kBatch = 4;   // 16-byte pieces per thread, and at a time
    uint4 gate[kBatch];
    const int otid = threadIdx.x - kSoftmax;
    auto load_gates = [&](int j0) {
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int i = (j0 + j) * 2 * kGroup + otid, r = i >> 5, c = i & 31;
        gate[j] = make_uint4(0, 0, 0, 0);
        if (p.gate != nullptr && r < n_rows)
          gate[j] = load_row16(p.gate + static_cast<long long>(t0 + r / G) * p.ld_gate + (kvh * G + r % G) * D + c * 8, wide);
      }
    };
    load_gates(0);
    asm volatile("bar.sync 4, 512;" ::: "memory");
#pragma unroll 1
    for (int j0 = 0; j0 < kOut && (j0 * 2 * kGroup >> 5) < n_rows; j0 += kBatch) {
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int i = (j0 + j) * 2 * kGroup + otid, r = i >> 5, c = i & 31;
        if (r >= n_rows) continue;
        uint4 o = *reinterpret_cast<const uint4*>(stage + r * kStagePitch + c * 16);
        if (p.gate != nullptr) {
          const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gate[j]);
          uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&ow[e]);
            ow[e] = pack_bf16x2(gate_by(__bfloat162float(v.x), __bfloat162float(g2[e].x)),
                                gate_by(__bfloat162float(v.y), __bfloat162float(g2[e].y)));
          }
        }
        store_row16(p.out + (static_cast<long long>(t0 + r / G) * p.n_q_heads + kvh * G + r % G) * D + c * 8, o, wide);
      }
      if (j0 + kBatch < kOut) load_gates(j0 + kBatch);
    }
  } else {
    // =========================== softmax: two threads per row = TMEM lane ===========================
    // Warps w and w + 4 share 32 rows: of every eight keys the first half takes the first four, the second the others, and
    // each half of the columns of Q and O.  (The row sum's four parts go by pairs of keys, so that each has two of them.)
    const int row = threadIdx.x & (kRows - 1), half = threadIdx.x / kRows;
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const auto row_bar = [&] { asm volatile("bar.sync %0, 64;" ::"r"(5 + (warp & 3)) : "memory"); };   // both halves of 32 rows
    // ---- this row of Q, (token row / G, head row % G), pre-scaled for exp2 softmax; rows past the block are zero ----
    if (n_tiles > 0) {
      const float qscale = p.sm_scale * 1.4426950408889634f;
      const __nv_bfloat16* src = p.q + (static_cast<long long>(t0 + row / G) * p.n_q_heads + kvh * G + row % G) * D;
#pragma unroll
      for (int c0 = 0; c0 < D / 2; c0 += 32) {
        const int c = half * (D / 2) + c0;
        uint4 raw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) raw[j] = row < n_rows ? load_row16(src + c + 8 * j, wide) : make_uint4(0, 0, 0, 0);
        uint32_t h[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
          for (int e = 0; e < 4; ++e) h[4 * j + e] = pack_half2(__bfloat162float(v[e].x) * qscale, __bfloat162float(v[e].y) * qscale);
        }
        tmem_st_x16(tmem + lane_sel + kColQ + c / 2, h);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars.p_full[1]));
    }
    // keys [lo, lim) are visible; rows past the block see everything (their results are not used)
    int lim = 0x7fffffff, lo = 0;
    if (row < n_rows) {
      lim = p.q_kv_len[t0 + row / G];
      if (p.window > 0) lo = max(0, lim - p.window);
    }
    // Scales of a tile: of the first half threads 0..63 fetch the K scales, 64..127 the V scales, the page two tiles and the
    // scale one tile ahead of their use.
    const int sv = row >> 6, skey = row & 63;
    int page_next = -1;
    uint32_t scale_raw = 0;    // fp8: the fp16 bits as loaded (decoded where they are used); mixed: the value's bits
    bool scale_live = false;
    PageWalk ask(k_first + skey, P), place = ask;
    int ask_key = k_first + skey;
    auto fetch_page = [&] {
      page_next = ask_key < k_end ? table[ask.page] : -1;
      ask_key += kKeys;
      ask.next_tile(P);
    };
    auto fetch_scale = [&] {
      const long long r = kv_row_of(p.kv, page_next, kvh, place.at);
      place.next_tile(P);
      scale_live = r >= 0;
      if (FORMAT == kKvFp8Row) {
        scale_raw = reinterpret_cast<const uint16_t*>(sv ? p.kv.v_scales : p.kv.k_scales)[scale_live ? r : 0];
      } else if (FORMAT == kKvMixed) {
        float f = 1.f;
        if (scale_live && kv_row_tier(r) == 1)
          f = __half2float(reinterpret_cast<const __half*>(sv ? p.kv.tier_v_scales[1] : p.kv.tier_k_scales[1])[kv_row_index(r)]);
        scale_raw = __float_as_uint(f);
      }
    };
    if (kScaled && half == 0 && n_tiles > 0) {
      fetch_page();
      fetch_scale();
      fetch_page();
    }
    float top = -CUDART_INF_F;   // the row's largest score so far
    // This half's two of the row sum's four parts: a row's parts are summed in key order whatever the block it is in.
    float l2[2] = {0.f, 0.f};
    for (int i = 0; i < n_tiles; ++i) {
      const int b = i & 1, kb = k_first + i * kKeys + half * 4;   // key of value j: kb + j / 4 * 8 + j % 4
      const float* ks = scale_s[b][0] + half * 4;
      const float* vs = scale_s[b][1] + half * 4;
      if constexpr (kScaled) {
        if (half == 0) {
          const float value = FORMAT == kKvFp8Row ? __half2float(__ushort_as_half(static_cast<unsigned short>(scale_raw))) : __uint_as_float(scale_raw);
          scale_s[b][sv][skey] = scale_live ? value : 0.f;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (half == 0) {
          fetch_scale();
          fetch_page();
        }
      }
      mbar_wait(smem_u32(&bars.s_full[b]), (i >> 1) & 1, abortp, p.status, kStatusPrefillWait);
      __syncwarp();
      tc_fence_after();
      const uint32_t s_addr = tmem + lane_sel + b * kKeys;
      // (nothing stands between a load from TMEM and its wait: the registers must not be touched, copied or spilled before)
      uint32_t v[kHalfKeys];
#pragma unroll
      for (int j = 0; j < kHalfKeys; j += 4) tmem_ld_x4(s_addr + 2 * j + half * 4, v + j);
      tmem_ld_wait_x32(v);
      // scores: scaled, keys out of sight at -inf
      if constexpr (kScaled) {
#pragma unroll
        for (int j = 0; j < kHalfKeys; j += 4) {
          const float4 k4 = *reinterpret_cast<const float4*>(ks + 2 * j);
          mul2(v[j], v[j + 1], k4.x, k4.y);
          mul2(v[j + 2], v[j + 3], k4.z, k4.w);
        }
      }
      if (!__all_sync(0xffffffffu, kb - half * 4 + kKeys <= lim && kb - half * 4 >= lo)) {
#pragma unroll
        for (int j = 0; j < kHalfKeys; ++j) {
          const int key = kb + j / 4 * 8 + j % 4;
          if (key >= lim || key < lo) v[j] = __float_as_uint(-CUDART_INF_F);
        }
      }
      float m4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) m4[j] = __uint_as_float(v[j]);
#pragma unroll
      for (int j = 4; j < kHalfKeys; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(v[j]));
      const float own = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      half_s[b][half][row] = own;
      // Both halves have their scores now, and either stores P over columns that the other has read: the fences put this warp's
      // loads from TMEM before the barrier and the other's stores behind it.
      tc_fence_before();
      row_bar();
      tc_fence_after();
      const float mx = fmaxf(own, half_s[b][half ^ 1][row]);
      const bool move = mx > top;
      const float corr = move ? ex2(top - mx) : 1.f;   // (a row's first keys: exp2(-inf) = 0)
      if (__any_sync(0xffffffffu, move)) {
        if (move) top = mx;
        if (i > 0) {
          mbar_wait(smem_u32(&bars.v_empty[b ^ 1]), ((i - 1) >> 1) & 1, abortp, p.status, kStatusPrefillWait);
          __syncwarp();
          tc_fence_after();
#pragma unroll 1
          for (int c = half * (D / 2); c < half * (D / 2) + D / 2; c += 32) {
            uint32_t o[32];
            tmem_ld_x32(tmem + lane_sel + kColO + c, o);
            tmem_ld_wait_x32(o);
#pragma unroll
            for (int j = 0; j < 32; j += 2) mul2(o[j], o[j + 1], corr, corr);
            tmem_st_x16(tmem + lane_sel + kColO + c, o);
            tmem_st_x16(tmem + lane_sel + kColO + c + 16, o + 16);
          }
        }
      }
      const float at = top == -CUDART_INF_F ? 0.f : top;   // (a row that has seen no key yet)
#pragma unroll
      for (int j = 0; j < kHalfKeys; j += 4) {
        float e[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) e[q] = __uint_as_float(v[j + q]);
        add2(e[0], e[1], -at, -at);
        add2(e[2], e[3], -at, -at);
#pragma unroll
        for (int q = 0; q < 4; ++q) e[q] = ex2(e[q]);
        if (j == 0) {   // (a part's first key of the tile)
          l2[0] = fmaf(l2[0], corr, e[0]);
          l2[1] = fmaf(l2[1], corr, e[2]);
        } else {
          add2(l2[0], l2[1], e[0], e[2]);
        }
        add2(l2[0], l2[1], e[1], e[3]);
        if constexpr (kScaled) {
          const float4 v4 = *reinterpret_cast<const float4*>(vs + 2 * j);
          e[0] *= v4.x; e[1] *= v4.y; e[2] *= v4.z; e[3] *= v4.w;
        }
        tmem_st_x2(s_addr + j + half * 2, pack_half2(e[0], e[1]), pack_half2(e[2], e[3]));
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars.p_full[b]));
    }
    // ---- normalised rows to the stage ----
    half_s[n_tiles & 1][half][row] = l2[0] + l2[1];
    if (n_tiles > 0) {
      mbar_wait(smem_u32(&bars.o_done), 0, abortp, p.status, kStatusPrefillWait);
      tc_fence_after();
    }
    row_bar();
    const float l = half_s[n_tiles & 1][0][row] + half_s[n_tiles & 1][1][row];
    const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
    for (int c = half * (D / 2); c < half * (D / 2) + D / 2; c += 32) {
      uint32_t o[32];
      if (n_tiles > 0) {
        tmem_ld_x32(tmem + lane_sel + kColO + c, o);
        tmem_ld_wait_x32(o);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = 0u;
      }
      uint4* dst = reinterpret_cast<uint4*>(stage + row * kStagePitch + c * 2);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = pack_bf16x2(__uint_as_float(o[8 * j + 2 * e]) * inv, __uint_as_float(o[8 * j + 2 * e + 1]) * inv);
        dst[j] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    asm volatile("bar.sync 4, 512;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kIssuer) tmem_dealloc(tmem, 512);
}

template <int FORMAT>
cudaError_t launch_fmt(const PrefillAttnParams& p, cudaStream_t stream, bool pdl) {
  auto kern = paged_attn_prefill_kernel<FORMAT>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.n_kv_heads, p.n_blocks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace

int prefill_attn_block_tokens(int n_q_heads, int n_kv_heads) {
  const int G = n_q_heads / n_kv_heads;
  return G > 0 && G <= kRows ? kRows / G : 0;
}

const char* paged_attention_prefill(const PrefillAttnParams& p, cudaStream_t stream, bool pdl) {
  if (p.n_blocks <= 0) return nullptr;
  if (p.head_dim != D) return "paged_attention_prefill: head_dim must be 256";
  if (p.n_q_heads % p.n_kv_heads) return "paged_attention_prefill: q heads must be a multiple of kv heads";
  if (p.kv.format == kKvInt8Group && (p.kv.group % 16)) return "paged_attention_prefill: int8 group must be a multiple of 16";
  cudaError_t e;
  switch (p.kv.format) {
    case kKvBf16: e = launch_fmt<kKvBf16>(p, stream, pdl); break;
    case kKvFp8Row: e = launch_fmt<kKvFp8Row>(p, stream, pdl); break;
    case kKvInt8Group: e = launch_fmt<kKvInt8Group>(p, stream, pdl); break;
    case kKvNvfp4: e = launch_fmt<kKvNvfp4>(p, stream, pdl); break;
    case kKvMixed: e = launch_fmt<kKvMixed>(p, stream, pdl); break;
    default: return "paged_attention_prefill: unknown KV format";
  }
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace nfb
