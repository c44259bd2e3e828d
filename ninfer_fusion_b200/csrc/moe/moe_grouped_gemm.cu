// Grouped expert GEMM for sm_100a: for every token tile of the expert-sorted receive buffer,
// out[rows, N_e] = x[rows, K] * W_e[N_e, K]^T with the expert taken from a device-side tile table.
//
// Same weight-stationary shape as the dense kernel (gemm_bf16.cu): 128 rows of W_e are the UMMA A operand, the tile's tokens
// the N operand, TMA -> 128B-swizzled shared memory -> tcgen05.mma -> TMEM -> tcgen05.ld epilogue.  A persistent CTA per SM
// walks (token tile, row tile) items; their number is read from the device, so the launch is graph-capturable although the
// routing is data dependent.  Warp 0 loads (a ring that runs on across items), warp 1 issues the products into two
// accumulators in turn, warps 2..9 drain them.  With one item per CTA the set-up of barriers and TMEM, the fill of the
// pipeline and the epilogue stood in the open: 2048 tokens, 256 experts of 1024 x 2048 and 2048 x 512, top-8 (1.07 and 0.54 GB
// of weights, 161 and 81 us at the copy rate) took 219 and 181 us.
// Epilogues:
//   gated unit (SwiGLU or a bounded form): W_e = [gate; up]; 64 gate rows + the matching 64 up rows form one 128-row tile;
//   return : each output row is stored into the return buffer of the rank that owns the token
//            (peer stores over NVLink), then that rank's arrival counter is advanced by the number
//            of rows it got from this CTA -- the combine all-to-all happens inside the GEMM.
//
// Reference: src/ops/sparse_moe/prefill/sparse_moe_prefill_kernels.cu (grouped mma.sync 64x64x64
// gate_up/down kernels after a select/scan/permute chain) and decode/sparse_moe_decode_kernels.cu.
#include "moe.h"

#include <cmath>
#include <mutex>
#include <unordered_map>

#include "../comm/peer_sync.cuh"
#include "../common/device.h"
#include "../common/launch.h"
#include "../common/ptx.cuh"
#include "../common/tensor_map.h"
#include "../gemm/persist_epilogue.cuh"

namespace nfb {

namespace {

constexpr int kBlockK = 64;
constexpr int kTileN = 128;
constexpr int kWTileBytes = kTileN * 128;

constexpr int kMaxTN = 256;
// Stages of the ring: a pair's of 24 KB fill the room; of one CTA's eight are enough, and with twelve small ones the weights come
// more slowly from memory (256 experts of 1024 x 2048, 16 rows each: 164 us, 155 with eight).
constexpr int kMaxStages = 12, kSingleStages = 8;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kSmemBytes = 221 * 1024;   // (4.5 KB of static tables beside it)
constexpr int kExchangeBytes = 4 * 2 * 2 * 8 * 32 * 4;   // gated unit: per warp pair two buffers x two directions x 8 x 32

struct MoeKernelParams {
  int tn;               // tokens per tile
  int n_row_tiles;      // row tiles per expert
  int num_kb;
  int rows_per_expert;  // N_e
  const int* tile_expert;
  const int* tile_row0;
  const int* tile_rows;
  const MoeState* state;
  __nv_bfloat16* out;
  long long ldo;
  int world;
  const int* recv_meta;
  __nv_bfloat16* peer_ret[kMoeMaxRanks];
  unsigned int* peer_ret_flag[kMoeMaxRanks];
  int* status;
  GluParams glu;
  // the dense expert: its items come first
  int dense_items, dense_tn, dense_row_tiles, dense_num_kb, dense_T, dense_rows;
  __nv_bfloat16* dense_out;
};

// Gated unit beside a dense expert (PAIR): the two CTAs of a cluster work on one item of twice the weight rows; each loads its own
// 128 rows and half of the tokens (see gemm_bf16.cu).  256 experts of 1024 x 2048, 2048 tokens, top-8: the dense expert's tokens
// beside them cost 3 us so and 16 with one CTA an item, whose shared memory they fill.  Without a dense expert the kernel is bound by
// the weights from HBM and one CTA an item is the faster or the same (us, pairs and one CTA: 16 rows an expert 162 and 155, 64 rows
// 179 and 177; 128 experts of 640 x 1024, whose third row tile leaves the second CTA idle, 33 and 31).  The return form has
// contractions of a few k-blocks, where handing an accumulator over between two CTAs shows (103 us, pairs 119).
// (token tile, row tile) of the walk
struct MoeItem {
  bool dense;
  int tile, xt;
};
__device__ __forceinline__ MoeItem moe_item(const MoeKernelParams& p, int item) {
  if (item < p.dense_items) return {true, item / p.dense_row_tiles, item % p.dense_row_tiles};
  item -= p.dense_items;
  return {false, item / p.n_row_tiles, item % p.n_row_tiles};
}

template <int EPI, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1) moe_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                               const __grid_constant__ CUtensorMap tmap_x,
                                                               const __grid_constant__ CUtensorMap tmap_dense_w,
                                                               const __grid_constant__ CUtensorMap tmap_dense_x,
                                                               const MoeKernelParams p) {
  constexpr int kRingBytes = kSmemBytes - 1024 - (EPI == kMoeEpiSwiglu ? kExchangeBytes : 0);
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages];
  __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
  __shared__ __align__(8) uint64_t bar_acc_full[2];
  __shared__ __align__(8) uint64_t bar_acc_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ __nv_bfloat16* dst_s[2][kMaxTN];  // return: where the rows of an item go
  __shared__ int src_cnt[2][kMoeMaxRanks];     // return, several ranks: rows of an item per source

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int TN = p.tn;
  const int crank = PAIR ? static_cast<int>(blockIdx.x & 1) : 0;
  const int walker = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int walkers = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  constexpr int kCtas = PAIR ? 2 : 1;
  const int stage_bytes = kWTileBytes + (p.dense_items > 0 ? max(TN, p.dense_tn) : TN) * 128 / kCtas;
  const int n_stages = min(PAIR ? kMaxStages : kSingleStages, kRingBytes / stage_bytes);
  const int half = p.rows_per_expert / 2;
  volatile int* abortp = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_acc_full[a]), 1);
      mbar_init(smem_u32(&bar_acc_empty[a]), (PAIR ? 2 : 1) * kEpiWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (threadIdx.x < 2 * kMoeMaxRanks) (&src_cnt[0][0])[threadIdx.x] = 0;
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(smem_u32(&tmem_base_slot), 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(&tmem_base_slot), 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // (the other CTA's barriers are initialised before anything counts on them)
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_launch_next();
  pdl_wait_prior();   // the tile table and the rows come from earlier kernels
  const int n_items = p.dense_items + p.state->n_tiles * p.n_row_tiles;

  if (warp == 0) {
    if (elect_one()) {
      // ---------------- TMA producer ----------------
      const uint64_t pol_w = l2_policy_evict_first();
      const uint64_t pol_x = l2_policy_evict_last();
      int s = 0;
      uint32_t ph = 1;      // the first pass over the ring finds every stage free
      uint32_t issued = 0;
      int item = walker;
      int expert = 0, row0 = 0;
      auto look_up = [&] {
        const MoeItem it = moe_item(p, item);
        if (item < n_items && !it.dense) {
          expert = p.tile_expert[it.tile];
          row0 = p.tile_row0[it.tile];
        }
      };
      look_up();
      while (item < n_items && !*abortp) {
        const MoeItem it = moe_item(p, item);
        const CUtensorMap* const map_w = it.dense ? &tmap_dense_w : &tmap_w;
        const CUtensorMap* const map_x = it.dense ? &tmap_dense_x : &tmap_x;
        const int wrow = it.dense ? 0 : expert * p.rows_per_expert;
        const int tn = it.dense ? p.dense_tn : TN;
        const int x_row = (it.dense ? it.tile * tn : row0) + crank * (tn / 2);
        const int row_a = wrow + (kCtas * it.xt + crank) * (EPI == kMoeEpiSwiglu ? 64 : kTileN);
        const int row_b = EPI == kMoeEpiSwiglu ? row_a + (it.dense ? p.dense_rows / 2 : half) : row_a + 64;
        const int num_kb = it.dense ? p.dense_num_kb : p.num_kb;
        const int bytes = kCtas * kWTileBytes + tn * 128;   // (of a pair, counted by the even CTA's barrier)
        item += walkers;
        look_up();   // the next item's entry, in flight beside this item's loads
        bool ok = true;
        for (int kb = 0; kb < num_kb; ++kb, ++issued) {
          if (!mbar_wait(smem_u32(&bar_empty[s]), ph, abortp, p.status, kStatusEmptyWaitTimeout)) {
            ok = false;
            break;
          }
          const uint32_t full = smem_u32(&bar_full[s]);
          const uint32_t dst = smem_base + s * stage_bytes;
          if (crank == 0) mbar_expect_tx(full, bytes);
          auto load = [&](uint32_t to, const CUtensorMap* map, int row, uint64_t pol) {
            if constexpr (PAIR) tma_load_2d_pair(to, map, mapa_shared(full, 0), kb * kBlockK, row, pol);
            else tma_load_2d(to, map, full, kb * kBlockK, row, pol);
          };
          load(dst, map_w, row_a, pol_w);
          load(dst + 64 * 128, map_w, row_b, pol_w);
          load(dst + kWTileBytes, map_x, x_row, pol_x);
          if (++s == n_stages) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
      }
      if (*abortp) {
        // Unwinding: let copies that were already issued land before the CTA exits.  (The odd CTA of a pair has no barrier
        // to see them by: its own never completes, and the polls are the pause.)
        const uint32_t depth = static_cast<uint32_t>(n_stages);
        for (uint32_t j = issued > depth ? issued - depth : 0; j < issued; ++j)
          for (uint32_t spin = 0; spin < (1u << 20); ++spin)
            if (mbar_try_wait(smem_u32(&bar_full[j % depth]), (j / depth) & 1)) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (crank == 0 && elect_one()) {
      // ---------------- MMA issuer (of both CTAs of a pair) ----------------
      int s = 0;
      uint32_t ph = 0;
      int n = 0;
      auto commit = [](uint32_t bar) {
        if constexpr (PAIR) tc_commit_pair(bar);
        else tc_commit(bar);
      };
      for (int item = walker; item < n_items && !*abortp; item += walkers, ++n) {
        const int a = n & 1;
        const bool dense = item < p.dense_items;
        const int num_kb = dense ? p.dense_num_kb : p.num_kb;
        const uint32_t idesc = umma_idesc(kCtas * kTileN, dense ? p.dense_tn : TN, 1, 1);
        // the epilogue has drained this accumulator's previous item
        if (n >= 2 && !mbar_wait(smem_u32(&bar_acc_empty[a]), ((n >> 1) & 1) ^ 1, abortp, p.status, kStatusAccumWaitTimeout)) break;
        tc_fence_after();
        const uint32_t acc = tmem_base + a * kMaxTN;
        bool ok = true;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&bar_full[s]), ph, abortp, p.status, kStatusTmaWaitTimeout)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_base + s * stage_bytes;
          const uint64_t a_desc = umma_desc_k_sw128(a_addr);
          const uint64_t b_desc = umma_desc_k_sw128(a_addr + kWTileBytes);
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k)
          {
            const uint32_t accumulate = (kb > 0 || k > 0) ? 1u : 0u;
            if constexpr (PAIR) tc_mma_f16_pair(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, accumulate);
            else tc_mma_f16(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, accumulate);
          }
          commit(smem_u32(&bar_empty[s]));
          if (++s == n_stages) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        commit(smem_u32(&bar_acc_full[a]));
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue warps ----------------
    const int etid = threadIdx.x - 64;
    const int lg = warp & 3;          // TMEM lane group this warp may read
    const int hf = (warp - 2) >> 2;   // which chunks of 16 tokens: hf, hf + 2, ...
    constexpr int kChunk = 16;
    float* const xch_s = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)) + kRingBytes);
    const int pair = (lg & 1) + 2 * hf;
    const uint32_t select = swap_select(lane);
    int n = 0, xch_i = 0;
    uint32_t returned = 0;            // one GPU: rows this CTA has returned
    for (int item = walker; item < n_items; item += walkers, ++n) {
      const MoeItem it = moe_item(p, item);
      const int row0 = it.dense ? it.tile * p.dense_tn : p.tile_row0[it.tile];
      const int rows = it.dense ? min(p.dense_tn, p.dense_T - row0) : p.tile_rows[it.tile];
      const int N = it.dense ? p.dense_rows : p.rows_per_expert;
      const int a = n & 1;
      if constexpr (EPI == kMoeEpiReturn) {
        if (etid < rows) {
          if (it.dense) {
            dst_s[a][etid] = p.dense_out + static_cast<long long>(row0 + etid) * N;
          } else {
            const int meta = p.recv_meta[row0 + etid];
            dst_s[a][etid] = p.peer_ret[meta >> 24] + static_cast<long long>(meta & 0xffffff) * N;
            if (p.world > 1) atomicAdd(&src_cnt[a][meta >> 24], 1);
          }
        }
      }
      const bool have = mbar_wait(smem_u32(&bar_acc_full[a]), (n >> 1) & 1, abortp, p.status, kStatusAccumWaitTimeout);
      // one verdict for the eight warps, so that the barriers below are never divergent
      if (!epi_all(have && !*abortp)) break;
      tc_fence_after();
      const uint32_t lane_taddr = tmem_base + a * kMaxTN + (static_cast<uint32_t>(lg * 32) << 16);
      if constexpr (EPI == kMoeEpiSwiglu) {
        // Lane groups 0, 1 hold gate rows, 2, 3 the matching up rows.  The two warps of a pair swap eight of a chunk's
        // sixteen columns, so that both finish half of the units.
        const bool is_up = lg >= 2;
        const int ne = ((kCtas * it.xt + crank) * 64 + (lg & 1) * 32 + lane) & ~1;
        __nv_bfloat16* const out = it.dense ? p.dense_out : p.out;
        const long long ldo = it.dense ? N / 2 : p.ldo;
        for (int c = hf * kChunk; c < rows; c += 2 * kChunk, ++xch_i) {
          float* buf = xch_s + (pair * 2 + (xch_i & 1)) * (2 * 8 * 32);
          float* mine = buf + (is_up ? 8 * 32 : 0);
          const float* other = buf + (is_up ? 0 : 8 * 32);
          uint32_t v[kChunk];
          tmem_ld_x16(lane_taddr + c, v);
          tmem_ld_wait_x16(v);
#pragma unroll
          for (int j = 0; j < 8; ++j) mine[j * 32 + lane] = __uint_as_float(is_up ? v[j] : v[8 + j]);
          epi_pair_sync(pair);
          const int cb = c + (is_up ? 8 : 0);
          uint32_t w[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            float o2[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int j = 2 * m + h;
              const float own = __uint_as_float(is_up ? v[8 + j] : v[j]);
              const float got = other[j * 32 + lane];
              o2[h] = gated_unit(is_up ? got : own, is_up ? own : got, p.glu);
            }
            const __nv_bfloat162 units = __floats2bfloat162_rn(o2[0], o2[1]);
            w[m] = swap_pair(*reinterpret_cast<const uint32_t*>(&units), select);
          }
          const int live = ne < N / 2 ? (rows - cb - (lane & 1) + 1) >> 1 : 0;
          store_rows<4>({out + static_cast<long long>(row0 + cb + (lane & 1)) * ldo + ne, 2 * ldo, live}, w);
        }
      } else {
        const int ne = ((kCtas * it.xt + crank) * kTileN + lg * 32 + lane) & ~1;
        for (int c = hf * kChunk; c < rows; c += 2 * kChunk) {
          uint32_t v[kChunk];
          tmem_ld_x16(lane_taddr + c, v);
          tmem_ld_wait_x16(v);
          __nv_bfloat16* const* dst = &dst_s[a][c + (lane & 1)];
          const int live = ne < N ? (rows - c - (lane & 1) + 1) >> 1 : 0;
#pragma unroll
          for (int m = 0; m < kChunk / 2; ++m) {
            const uint32_t w = swap_pair(pack_bf16x2(__uint_as_float(v[2 * m]), __uint_as_float(v[2 * m + 1])), select);
            if (m < live) *reinterpret_cast<uint32_t*>(dst[2 * m] + ne) = w;
          }
        }
      }
      // this warp is done with the accumulator: hand it back to the MMA issuer
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&bar_acc_empty[a]), 0));
        else mbar_arrive(smem_u32(&bar_acc_empty[a]));
      }
      if constexpr (EPI == kMoeEpiReturn) {
        // One arrival unit per returned row of a 128-column tile.  Several ranks: signalled per item, so that the owners can
        // start early (the barrier orders all stores before the signalling threads, whose system-scope fence + release is
        // cumulative over them).  One GPU: the kernel's end orders the stores, the counter is advanced once per CTA.
        if (p.world == 1) {
          if (!it.dense) returned += static_cast<uint32_t>(rows);
        } else {
          epi_all(true);
          if (etid < p.world) {
            const int cnt = src_cnt[a][etid];
            src_cnt[a][etid] = 0;   // (filled again two items on, behind that item's predecessor's barriers)
            if (cnt > 0) {
              __threadfence_system();
              red_release_sys_add(p.peer_ret_flag[etid], static_cast<uint32_t>(cnt));
            }
          }
        }
      }
    }
    if constexpr (EPI == kMoeEpiReturn) {
      if (p.world == 1) {
        __threadfence();
        if (epi_all(true) && etid == 0 && returned > 0 && !*abortp) red_release_gpu_add(p.peer_ret_flag[0], returned);
      }
    }
  }

  tc_fence_before();
  if constexpr (PAIR) {
    cluster_sync_all();   // (the other CTA neither reads this one's operands nor arrives on its barriers any more)
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
  } else {
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
  }
}

template <int EPI, bool PAIR>
cudaError_t launch(const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& dw, const CUtensorMap& dx,
                   const MoeKernelParams& kp, long long max_items, cudaStream_t stream, bool pdl) {
  auto kern = moe_gemm_kernel<EPI, PAIR>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  constexpr int kCtas = PAIR ? 2 : 1;
  const long long walkers = device_sm_count() / kCtas;
  const dim3 grid(static_cast<unsigned>(kCtas * (max_items < walkers ? max_items : walkers)));
  return launch_kernel(kern, grid, dim3(kThreads), kSmemBytes, stream, pdl, kCtas, tw, tx, dw, dx, kp);
}

struct Key {
  const void* base; uint64_t rows, cols, ld; uint32_t box;
  bool operator==(const Key& o) const { return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box == o.box; }
};
struct KeyHash {
  size_t operator()(const Key& k) const {
    size_t h = reinterpret_cast<size_t>(k.base);
    h = h * 1000003u ^ k.rows; h = h * 1000003u ^ k.cols; h = h * 1000003u ^ k.ld;
    return h * 1000003u ^ k.box;
  }
};
bool cached_tmap(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box) {
  static std::mutex mu;
  static std::unordered_map<Key, CUtensorMap, KeyHash> cache;
  Key key{base, rows, cols, ld, box};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return true; }
  CUtensorMap m;
  if (!make_tmap_2d(&m, TmapDtype::BF16, base, rows, cols, ld, box, kBlockK, true)) return false;
  if (cache.size() > 65536) cache.clear();
  cache.emplace(key, m);
  *out = m;
  return true;
}

}  // namespace

int moe_tile_tokens(double rows_per_expert) {
  if (rows_per_expert <= 16) return 16;
  if (rows_per_expert <= 32) return 32;
  if (rows_per_expert <= 64) return 64;
  if (rows_per_expert <= 160) return 128;
  return 256;
}

// Wide enough for nearly every expert when tokens choose experts at random (mean + 2.5 standard deviations), so that its
// weights are streamed once; a mean of 64 rows in tiles of 64 made every other expert a second tile of a few rows.  More than
// 256 are shared out evenly.
int moe_token_tile(double rows_per_expert) {
  const double want = rows_per_expert + 2.5 * sqrt(rows_per_expert > 0 ? rows_per_expert : 0.);
  const int n = static_cast<int>(ceil(want / kMaxTN));
  const int tn = (static_cast<int>(ceil(want / (n < 1 ? 1 : n))) + 15) / 16 * 16;
  return tn < 16 ? 16 : (tn > kMaxTN ? kMaxTN : tn);
}

const char* moe_gemm(const MoeGemmArgs& a) {
  if (a.n_local_experts <= 0 || a.rows_per_expert <= 0 || a.K <= 0 || a.cap <= 0) return "moe_gemm: empty problem";
  if ((a.K % 8) || (a.ldw % 8) || (a.ldx % 8)) return "moe_gemm: K and leading dims must be multiples of 8";
  if ((reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.x)) & 15) return "moe_gemm: operands must be 16-byte aligned";
  const int tn = a.tile_tokens;
  if (tn < 16 || tn > kMaxTN || tn % 16) return "moe_gemm: bad token tile";
  if (a.max_tiles < 1 || a.max_tiles > 65535) return "moe_gemm: tile bound out of range";
  if (a.tile_expert == nullptr || a.tile_row0 == nullptr || a.tile_rows == nullptr || a.state == nullptr)
    return "moe_gemm: missing tile table";
  MoeKernelParams kp = {};
  kp.num_kb = static_cast<int>((a.K + kBlockK - 1) / kBlockK);
  kp.rows_per_expert = static_cast<int>(a.rows_per_expert);
  kp.tile_expert = a.tile_expert; kp.tile_row0 = a.tile_row0; kp.tile_rows = a.tile_rows; kp.state = a.state;
  kp.status = a.status; kp.glu = a.glu;
  kp.tn = tn;
  const bool swiglu = a.epi == kMoeEpiSwiglu, pair = swiglu && a.dense_w != nullptr;
  const int ctas = pair ? 2 : 1;
  if (swiglu) {
    if (a.rows_per_expert % 128) return "moe_gemm: SwiGLU needs expert rows in multiples of 128 (64 gate + 64 up per tile)";
    if (a.out == nullptr || (a.ldo & 1)) return "moe_gemm: no output";
    kp.out = static_cast<__nv_bfloat16*>(a.out); kp.ldo = a.ldo;
    kp.n_row_tiles = static_cast<int>((a.rows_per_expert / 2 + 64 * ctas - 1) / (64 * ctas));
  } else if (a.epi == kMoeEpiReturn) {
    if (a.rows_per_expert % 8) return "moe_gemm: expert rows must be a multiple of 8";
    if (a.world < 1 || a.world > kMoeMaxRanks || a.recv_meta == nullptr) return "moe_gemm: bad return set-up";
    kp.world = a.world; kp.recv_meta = a.recv_meta;
    for (int r = 0; r < a.world; ++r) {
      if (a.peer_ret[r] == nullptr || a.peer_ret_flag[r] == nullptr) return "moe_gemm: missing peer pointer";
      kp.peer_ret[r] = a.peer_ret[r]; kp.peer_ret_flag[r] = a.peer_ret_flag[r];
    }
    kp.n_row_tiles = static_cast<int>((a.rows_per_expert + 127) / 128);
  } else {
    return "moe_gemm: unknown epilogue";
  }
  CUtensorMap tw, tx;
  if (!cached_tmap(&tw, a.w, static_cast<uint64_t>(a.n_local_experts) * a.rows_per_expert, a.K, a.ldw, 64))
    return "moe_gemm: weight tensor map rejected";
  if (!cached_tmap(&tx, a.x, a.cap, a.K, a.ldx, tn / ctas)) return "moe_gemm: activation tensor map rejected";
  CUtensorMap dw = tw, dx = tx;
  if (a.dense_w != nullptr) {
    if (a.dense_x == nullptr || a.dense_out == nullptr || a.dense_T <= 0 || a.dense_K <= 0 || a.dense_K % 8 ||
        a.dense_rows <= 0 || a.dense_rows % (swiglu ? 128 : 8))
      return "moe_gemm: bad dense expert";
    if ((reinterpret_cast<uintptr_t>(a.dense_w) | reinterpret_cast<uintptr_t>(a.dense_x)) & 15 || reinterpret_cast<uintptr_t>(a.dense_out) & 3)
      return "moe_gemm: dense operands must be 16-byte aligned";
    // its own token tile: the routed one follows the few rows of an expert, and 128 tokens of a pair or 64 fit eight stages
    const int few = static_cast<int>((a.dense_T + 15) / 16 * 16), wide = 64 * ctas;
    kp.dense_tn = tn > wide ? tn : (few < wide ? (few > tn ? few : tn) : wide);
    kp.dense_T = static_cast<int>(a.dense_T);
    kp.dense_rows = static_cast<int>(a.dense_rows);
    kp.dense_num_kb = static_cast<int>((a.dense_K + kBlockK - 1) / kBlockK);
    kp.dense_row_tiles = swiglu ? (kp.dense_rows / 2 + 64 * ctas - 1) / (64 * ctas) : (kp.dense_rows + kTileN - 1) / kTileN;
    kp.dense_items = kp.dense_row_tiles * ((kp.dense_T + kp.dense_tn - 1) / kp.dense_tn);
    kp.dense_out = a.dense_out;
    if (!cached_tmap(&dw, a.dense_w, a.dense_rows, a.dense_K, a.dense_K, 64)) return "moe_gemm: dense weight tensor map rejected";
    if (!cached_tmap(&dx, a.dense_x, a.dense_T, a.dense_K, a.dense_K, kp.dense_tn / ctas)) return "moe_gemm: dense activation tensor map rejected";
  }
  const long long max_items = static_cast<long long>(a.max_tiles) * kp.n_row_tiles + kp.dense_items;
  cudaError_t e = !swiglu ? launch<kMoeEpiReturn, false>(tw, tx, dw, dx, kp, max_items, a.stream, a.pdl)
                  : pair  ? launch<kMoeEpiSwiglu, true>(tw, tx, dw, dx, kp, max_items, a.stream, a.pdl)
                          : launch<kMoeEpiSwiglu, false>(tw, tx, dw, dx, kp, max_items, a.stream, a.pdl);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace nfb
