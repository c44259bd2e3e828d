// Weight-stationary bf16 GEMM for sm_100a:  out[T, N] = x[T, K] * W[N, K]^T.
//
// The weight matrix is the UMMA "A" operand (M = 128 weight rows per CTA), the
// activations are the "B" operand (UMMA N = TN tokens, 16..256), so one kernel
// template covers decode (T = 1..64: pure weight streaming) and prefill
// (T tiles of 256).  Operands arrive by TMA into 128-byte-swizzled shared
// memory, tcgen05.mma accumulates in TMEM, and the epilogue reads TMEM with
// tcgen05.ld and fuses: plain store (+bias), residual add, SwiGLU (gate and up
// rows of the fused [gate; up] parent are loaded as two 64-row boxes of one
// 128-row tile), or fp32 split-K partials.
//
// Covers the reference's linear / linear_add / linear_swiglu bf16 routes
// (include/ninfer/ops/linear.h, src/ops/linear/bf16/bf16_gemm_mma.cuh,
// src/ops/linear_swiglu/*, src/ops/linear_add/*), which are mma.sync kernels.
#include "gemm.h"

#include <mutex>
#include <unordered_map>

#include <cstdlib>

#include "../comm/peer_sync.cuh"
#include "../common/device.h"
#include "../common/ptx.cuh"
#include "../common/tensor_map.h"
#include "persist_epilogue.cuh"

namespace nfb {

namespace {

constexpr int kBlockK = 64;           // bf16 elements per k-block = one 128-byte swizzle row
constexpr int kTileN = 128;           // weight rows per CTA (UMMA M)
constexpr int kWTileBytes = kTileN * 128;

// DEEP = one CTA per SM with a pipeline twice as deep: used when the whole grid fits in one wave, so that a
// grid of ~100 CTAs still keeps ~200 KB per SM in flight (the memory system needs ~30 MB in flight overall).
template <int TN, bool DEEP = false>
struct GemmCfg {
  // Plain epilogues above 32 tokens take the persistent kernel; TN = 128 and 256 serve the split, gathered and peer epilogues.
  // TN = 256: the main loop runs at the tensor rate, so what matters is hiding the epilogue.  Two stages = 96 KB let two CTAs share
  // an SM (and its 512 TMEM columns): one drains its accumulator while the other feeds the tensor core.  A grid that fits in one
  // wave keeps the four-stage pipeline (DEEP).
  static constexpr int kStages =
      DEEP ? (TN <= 32 ? 10 : (TN == 256 ? 4 : 8)) : (TN <= 32 ? 5 : (TN == 64 ? 4 : (TN == 128 ? 6 : 2)));
  static constexpr int kXTileBytes = TN * 128;
  static constexpr int kStageBytes = kWTileBytes + kXTileBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024;  // +1024: manual alignment
  static constexpr int kTmemCols = TN < 32 ? 32 : TN;
};

// Optional phase timeline (globaltimer, ns) of every CTA, for performance debugging: 8 stamps per CTA.
constexpr int kTraceStamps = 12;
constexpr int kTraceCtas = 4096;
__device__ unsigned long long g_gemm_trace[kTraceCtas * kTraceStamps];
bool g_trace_enabled = false;
// Timeline over SEVERAL launches (a whole layer, a captured graph): launch i of a traced run writes the stamps of
// its first kTimelineCtas CTAs into slot i % kTimelineSlots, so that the overlap of consecutive kernels under
// programmatic dependent launch can be read off one clock (globaltimer).
constexpr int kTimelineSlots = 64;
constexpr int kTimelineCtas = 256;
__device__ unsigned long long g_gemm_timeline[kTimelineSlots * kTimelineCtas * kTraceStamps];
int g_timeline_next = -1;   // < 0: off; else the slot of the next launch

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

struct KernelParams {
  int trace;
  int T, N, K;
  int tn;              // persistent kernel: tokens per tile
  int kb_per_split;    // k-blocks handled by one blockIdx.z
  int num_kb;          // ceil(K / 64)
  int swiglu_half;     // N/2 for the SwiGLU epilogue, else 0
  GluParams glu;
  __nv_bfloat16* out;
  long long ldo;
  const __nv_bfloat16* resid;
  long long ldr;
  const float* bias;
  int act;  // GemmActivation, applied after the bias (kEpiStore only)
  const float* act_params;
  float* out32;        // kEpiStore: columns >= out32_from as fp32 (nullptr: none)
  long long ldo32;
  int out32_from;
  float* partial;      // [splits, T, N] fp32
  int* status;
  // kEpiPushPartial: tensor-parallel reduce-scatter by peer stores
  float* peer_recv[kMaxRanks];
  unsigned int* peer_flag[kMaxRanks];
  int rank, slice_cols;
  // in-cluster split-K: `cluster` CTAs along z share one output tile and reduce through DSMEM
  int cluster;
  // kEpiPushAll: one-shot all-reduce by push into [parity][src_rank][T_cap][N] on every rank
  int world, T_cap;
  const unsigned int* call_idx;  // device counter of finished reduce calls; its parity picks the buffer
  // kEpiRsAg: reduce-scatter into the owner, owner-side reduction, all-gather of the new residual tile
  __nv_bfloat16* peer_x[kMaxRanks];
  long long ld_resid;
  float* peer_ss[kMaxRanks];
  unsigned int* peer_xflag[kMaxRanks];
  uint2* peer_recv_ll[kMaxRanks];   // [src][T_cap][N / world] (fp32 bits, epoch)
  RsState* rs_state;
  int rs_phase;
  // gathered consumer (kEpiStore / kEpiSwiglu): wait for the residual tiles, RMS norm as an epilogue row scale
  const unsigned int* g_flag;
  const unsigned int* g_target;
  const float* g_ss;
  int g_tiles;
  float g_inv_n, g_eps;
  // kEpiStore: decode conv + SiLU + history roll on columns [0, conv_C)
  const __nv_bfloat16* conv_w;
  __nv_bfloat16* conv_state;
  const int* conv_slot;
  __nv_bfloat16* conv_out;
  int conv_C;
  // L2 prefetch hint for the next kernel's weights: each CTA asks for `pf_per_cta` bytes of [pf_ptr, pf_ptr + pf_bytes)
  const uint8_t* pf_ptr;
  long long pf_bytes;
  int pf_per_cta;
};

// GELU in the two forms vision towers use: tanh approximation (transformer blocks) and exact erf (merger).
__device__ __forceinline__ float gelu(float x, int mode) {
  if (mode == kActGeluTanh) {
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return 0.5f * x * (1.f + tanhf(u));
  }
  return 0.5f * x * (1.f + erff(x * 0.7071067811865476f));
}

__device__ __forceinline__ float activate(float z, int mode, float a, float b) {
  if (mode == kActXielu)
    return z > 0.f ? (a * z + 0.5f) * z : b * (__expf(z) - 1.f - z) + 0.5f * z;
  if (mode == kActRelu2) return z > 0.f ? z * z : 0.f;
  if (mode == kActSoftcap) return a * tanhf(z * b);
  return gelu(z, mode);
}

template <int TN, int EPI, bool DEEP>
__global__ void __launch_bounds__(128) gemm_ws_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                       const __grid_constant__ CUtensorMap tmap_x,
                                                       const KernelParams p) {
  using Cfg = GemmCfg<TN, DEEP>;
  constexpr int kStages = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kStages];
  __shared__ __align__(8) uint64_t bar_empty[kStages];
  __shared__ __align__(8) uint64_t bar_accum;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int peer_ok[kMaxRanks];
  __shared__ float row_s[TN];   // per token: RMS factor (gathered consumer) or the tile's sum of squares (kEpiRsAg)
  __shared__ int rs_ok;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int cta_linear = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  auto stamp = [&](int i) {
    if (p.trace && threadIdx.x == 0) {
      const unsigned long long now = globaltimer_ns();
      if (cta_linear < kTraceCtas) g_gemm_trace[cta_linear * kTraceStamps + i] = now;
      if (p.trace > 1 && cta_linear < kTimelineCtas)
        g_gemm_timeline[((p.trace - 2) * kTimelineCtas + cta_linear) * kTraceStamps + i] = now;
    }
  };
  stamp(0);

  const int t0 = blockIdx.y * TN;
  const int n0 = (EPI == kEpiSwiglu) ? blockIdx.x * 64 : blockIdx.x * kTileN;
  const int kb_begin = blockIdx.z * p.kb_per_split;
  const int kb_end = min(p.num_kb, kb_begin + p.kb_per_split);
  // (phase 2 of kEpiRsAg runs no GEMM: the tiles were left in the receive buffers by phase 1)
  const int num_it = (EPI == kEpiRsAg && p.rs_phase == 2) ? 0 : kb_end - kb_begin;
  const bool gathered = (EPI == kEpiStore || EPI == kEpiSwiglu) && p.g_flag != nullptr;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int r = 0; r < kMaxRanks; ++r) peer_ok[r] = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_accum), 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(&tmem_base_slot), Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  stamp(1);

  // Let the next kernel in the stream begin its own prologue / weight prefetch.
  pdl_launch_next();

  if (warp == 0) {
    if (elect_one()) {
      // ---------------- TMA producer ----------------
      const uint64_t pol_w = l2_policy_evict_first();
      const uint64_t pol_x = l2_policy_evict_last();
      const int row_a = n0;
      const int row_b = (EPI == kEpiSwiglu) ? p.swiglu_half + n0 : n0 + 64;
      // Weights do not depend on the previous kernel: fill EVERY stage with them before waiting for it, so that the
      // whole pipeline (not one stage) is in flight while the previous kernel drains.  Only then the activations:
      // after the previous kernel (plain input), or after the owner ranks have pushed their residual tiles into
      // this rank's buffer (gathered input; bounded wait).
      const int pre = num_it < kStages ? num_it : kStages;
      for (int j = 0; j < pre; ++j) {
        const uint32_t full = smem_u32(&bar_full[j]);
        const uint32_t dst = smem_base + j * Cfg::kStageBytes;
        const int kx = (kb_begin + j) * kBlockK;
        mbar_expect_tx(full, Cfg::kStageBytes);
        tma_load_2d(dst, &tmap_w, full, kx, row_a, pol_w);
        tma_load_2d(dst + 64 * 128, &tmap_w, full, kx, row_b, pol_w);
      }
      pdl_wait_prior();
      if (gathered) {
        const uint32_t target = __ldcg(p.g_target);
        // on a time-out the loads below are still issued (the data is stale, the status word says so): every
        // barrier that was armed above must complete before the CTA may leave
        if (!wait_counter(p.g_flag, target, p.status)) abort_flag = 1;
        asm volatile("fence.proxy.async.global;" ::: "memory");
      }
      for (int j = 0; j < pre; ++j)
        tma_load_2d(smem_base + j * Cfg::kStageBytes + kWTileBytes, &tmap_x, smem_u32(&bar_full[j]),
                    (kb_begin + j) * kBlockK, t0, pol_x);
      int it = pre;
      for (; it < num_it; ++it) {
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1;
        if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1, &abort_flag, p.status, kStatusEmptyWaitTimeout)) break;
        const uint32_t full = smem_u32(&bar_full[s]);
        const uint32_t dst = smem_base + s * Cfg::kStageBytes;
        const int kx = (kb_begin + it) * kBlockK;
        mbar_expect_tx(full, Cfg::kStageBytes);
        tma_load_2d(dst, &tmap_w, full, kx, row_a, pol_w);
        tma_load_2d(dst + 64 * 128, &tmap_w, full, kx, row_b, pol_w);
        tma_load_2d(dst + kWTileBytes, &tmap_x, full, kx, t0, pol_x);
      }
      if (abort_flag) {
        // Unwinding: let copies that were already issued land before the CTA exits.
        const int first = it > kStages ? it - kStages : 0;
        for (int j = first; j < it; ++j) {
          const uint32_t bar = smem_u32(&bar_full[j % kStages]);
          const uint32_t ph = (j / kStages) & 1;
          for (uint32_t spin = 0; spin < (1u << 20); ++spin)
            if (mbar_try_wait(bar, ph)) break;
        }
      } else if (p.pf_per_cta > 0) {
        // own loads are all in flight: pull this CTA's share of the next kernel's weights into L2
        const long long off = static_cast<long long>(cta_linear) * p.pf_per_cta;
        if (off < p.pf_bytes) {
          const long long n = min(static_cast<long long>(p.pf_per_cta), p.pf_bytes - off) & ~15LL;
          if (n > 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.pf_ptr + off), "r"(static_cast<uint32_t>(n))
                         : "memory");
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc = umma_idesc(kTileN, TN, 1, 1);
      bool ok = true;
      for (int it = 0; it < num_it; ++it) {
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1;
        if (!mbar_wait(smem_u32(&bar_full[s]), ph, &abort_flag, p.status, kStatusTmaWaitTimeout)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_addr = smem_base + s * Cfg::kStageBytes;
        const uint64_t a_desc = umma_desc_k_sw128(a_addr);
        const uint64_t b_desc = umma_desc_k_sw128(a_addr + kWTileBytes);
#pragma unroll
        for (int k = 0; k < kBlockK / 16; ++k) {
          // advance 16 elements (32 bytes) along K inside the swizzle atom: +2 in 16-byte units
          tc_mma_f16(tmem_base, a_desc + 2 * k, b_desc + 2 * k, idesc, (it > 0 || k > 0) ? 1u : 0u);
        }
        tc_commit(smem_u32(&bar_empty[s]));
      }
      if (ok) tc_commit(smem_u32(&bar_accum));
    }
    __syncwarp();
  }

  // ---------------- epilogue: all four warps, warp w owns TMEM lanes 32w..32w+31 ----------------
  pdl_wait_prior();
  // kEpiRsAg: the bookkeeping word of this CTA's tile (its epoch) is fetched now, so that the latency hides under
  // the main loop
  uint32_t epoch_pre = 0;
  if constexpr (EPI == kEpiRsAg) {
    if (p.cluster <= 1 || blockIdx.z == 0) epoch_pre = p.rs_state->tile_epoch[blockIdx.x * kRsMaxTokenTiles + blockIdx.y];
  }
  if constexpr (EPI == kEpiStore) {
    // decode conv tiles: pull this thread's history columns towards L2 now (fire and forget), so that the
    // dependent slot -> history loads of the epilogue do not each pay a trip to HBM after the main loop
    if (p.conv_state != nullptr && n0 < p.conv_C && (p.cluster <= 1 || blockIdx.z == 0)) {
      const int n = n0 + threadIdx.x;
      for (int t = t0; t < min(p.T, t0 + TN); ++t) {
        const __nv_bfloat16* st = p.conv_state + static_cast<long long>(p.conv_slot[t]) * 3 * p.conv_C + n;
        if ((threadIdx.x & 31) == 0) {   // one request per 64-byte run of a warp's channels
#pragma unroll
          for (int j = 0; j < 3; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(st + j * p.conv_C));
        }
      }
    }
  }
  bool have_acc = true;
  if (num_it > 0) {
    have_acc = mbar_wait(smem_u32(&bar_accum), 0, &abort_flag, p.status, kStatusAccumWaitTimeout);
  }
  tc_fence_after();
  // One CTA-wide verdict, so the barriers inside the epilogue are never divergent.
  int epilogue_ok = __syncthreads_and(have_acc && !abort_flag);
  stamp(2);
  const uint32_t lane_taddr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
  constexpr int kChunk = 16;

  // ---------------- in-cluster split-K: peers hand their fp32 tiles to the leader through DSMEM ----------------
  const int S = p.cluster;
  const uint32_t crank = S > 1 ? blockIdx.z : 0;
  // leader-side landing zone in the (now idle) pipeline stages: [S-1][TN][128] floats
  const float* peer_s = reinterpret_cast<const float*>(smem_raw + (smem_base - smem_u32(smem_raw)));
  if (S > 1) {
    // #1: every CTA of the cluster has retired its MMAs, so the leader's stages may be overwritten
    cluster_sync_all();
    if (crank != 0) {
      if (epilogue_ok) {
        const uint32_t local = smem_base + ((crank - 1) * TN * 128 + warp * 32 + lane) * 4;
        const uint32_t remote = mapa_shared(local, 0);
        for (int c = 0; c < TN; c += kChunk) {
          uint32_t v[kChunk];
          tmem_ld_x16(lane_taddr + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kChunk; ++j) st_shared_cluster_u32(remote + (c + j) * 512, num_it > 0 ? v[j] : 0u);
        }
      }
      if (threadIdx.x == 0) st_shared_cluster_u32(mapa_shared(smem_u32(&peer_ok[crank]), 0), epilogue_ok ? 1u : 0u);
    }
    stamp(3);
    // #2: peers' tiles (release) are visible to the leader (acquire)
    cluster_sync_all();
    stamp(4);
    if (crank != 0) {
      epilogue_ok = 0;  // only the leader writes the output
    } else {
      for (int r = 1; r < S; ++r) epilogue_ok &= peer_ok[r];
    }
  }
  if (gathered) {
    // RMS factor of every token of the tile from the per-tile sums of squares that travelled with the residual
    if (threadIdx.x == 0) (void)ld_acquire_sys(p.g_flag);
    __syncthreads();
    for (int t = threadIdx.x; t < TN; t += 128) {
      // the whole table row in independent 16-byte loads (entries past the last tile are never written: zero)
      float ss = 0.f;
      if (t0 + t < p.T) {
        const float4* rowp = reinterpret_cast<const float4*>(p.g_ss + static_cast<long long>(t0 + t) * kRsSsStride);
        float4 q[kRsSsStride / 4];
#pragma unroll
        for (int j = 0; j < kRsSsStride / 4; ++j) q[j] = __ldcg(rowp + j);
#pragma unroll
        for (int j = 0; j < kRsSsStride / 4; ++j) ss += (q[j].x + q[j].y) + (q[j].z + q[j].w);
      }
      row_s[t] = rsqrtf(ss * p.g_inv_n + p.g_eps);
    }
    __syncthreads();
  }
  // accumulator chunk = own TMEM columns + the peers' contributions, summed in rank order
  auto load_acc = [&](int c, float* acc) {
    uint32_t v[kChunk];
    tmem_ld_x16(lane_taddr + c, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < kChunk; ++j) acc[j] = num_it > 0 ? __uint_as_float(v[j]) : 0.f;
    for (int r = 1; r < S; ++r) {
#pragma unroll
      for (int j = 0; j < kChunk; ++j) acc[j] += peer_s[((r - 1) * TN + c + j) * 128 + warp * 32 + lane];
    }
    if (gathered) {
#pragma unroll
      for (int j = 0; j < kChunk; ++j) acc[j] *= row_s[c + j];
    }
  };

  if (epilogue_ok) {
    if constexpr (EPI == kEpiSwiglu) {
      // lanes 0..63 hold gate rows, lanes 64..127 the matching up rows.
      float* up_s = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw))) +
                    (S - 1) * TN * 128;  // [TN][64], behind the peers' landing zone
      if (warp >= 2) {
        const int r = (warp - 2) * 32 + lane;
        for (int c = 0; c < TN; c += kChunk) {
          float v[kChunk];
          load_acc(c, v);
#pragma unroll
          for (int j = 0; j < kChunk; ++j) up_s[(c + j) * 64 + r] = v[j];
        }
      }
      __syncthreads();
      if (warp < 2) {
        const int r = warp * 32 + lane;
        const int n = n0 + r;
        for (int c = 0; c < TN; c += kChunk) {
          float v[kChunk];
          load_acc(c, v);
#pragma unroll
          for (int m = 0; m < kChunk / 2; ++m) {
            float a[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int j = 2 * m + h;
              const float g = v[j];
              const float u = up_s[(c + j) * 64 + r];
              a[h] = gated_unit(g, u, p.glu);
            }
            const float send = (lane & 1) ? a[0] : a[1];
            const float recv = __shfl_xor_sync(0xffffffffu, send, 1);
            const int t = t0 + c + 2 * m + (lane & 1);
            const int ne = n & ~1;
            if (t < p.T && ne < p.swiglu_half) {
              const uint32_t packed = (lane & 1) ? pack_bf16x2(recv, a[1]) : pack_bf16x2(a[0], recv);
              *reinterpret_cast<uint32_t*>(p.out + static_cast<long long>(t) * p.ldo + ne) = packed;
            }
          }
        }
      }
    } else if constexpr (EPI == kEpiPushPartial) {
      // reduce-scatter by push: this tile's columns belong to one owner rank; the fp32 partial goes into the
      // owner's receive buffer [src_rank][split][T][slice_cols].  The tile passes through shared memory (the idle
      // pipeline stages), up to 128 token rows at a time, so that the stores are 16 bytes wide and every token row
      // of the tile is one contiguous 512-byte run, instead of 4-byte stores in 128-byte runs.
      const int owner = n0 / p.slice_cols;
      constexpr int kRowPad = kTileN + 4;
      constexpr int kRows = TN < 128 ? TN : 128;
      float* tile_s = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));
      const int col = (threadIdx.x & 3) * 32;
      float* dst = p.peer_recv[owner] + (static_cast<long long>(p.rank) * gridDim.z + blockIdx.z) * p.T * p.slice_cols +
                   (n0 + col - owner * p.slice_cols);
      for (int h = 0; h < TN; h += kRows) {
        if (t0 + h >= p.T) break;
        for (int c = h; c < h + kRows; c += kChunk) {
          if (t0 + c >= p.T) break;
          float v[kChunk];
          load_acc(c, v);
#pragma unroll
          for (int j = 0; j < kChunk; ++j) tile_s[(c - h + j) * kRowPad + warp * 32 + lane] = v[j];
        }
        __syncthreads();
        for (int r = threadIdx.x >> 2; r < kRows; r += 32) {
          const int t = t0 + h + r;
          if (t >= p.T) continue;
          const float4* src4 = reinterpret_cast<const float4*>(tile_s + r * kRowPad + col);
          float4* dst4 = reinterpret_cast<float4*>(dst + static_cast<long long>(t) * p.slice_cols);
#pragma unroll
          for (int q = 0; q < 8; ++q) dst4[q] = src4[q];
        }
        __syncthreads();   // (orders the peer stores before the signalling thread; frees the staging tile)
      }
      // publish: the signalling thread's release (system scope) is cumulative over the stores the barrier ordered
      if (threadIdx.x == 0) red_release_sys_add(p.peer_flag[owner], 1u);
    } else if constexpr (EPI == kEpiRsAg) {
      const int owner = n0 / p.slice_cols;
      const bool pushes = p.rs_phase != 2;
      const bool reduces = p.rs_phase != 1;
      // Every call of this tile carries the next epoch: the tile's fp32 values travel as (value, epoch) pairs, so
      // the reader sees from the data itself when a tile is complete.  No fence and no counter sit between the
      // writer's stores and the reader's loads (16-byte stores are not torn).  Every tile of one state object is
      // written once per call, so all tiles carry the same epoch.
      unsigned int* epoch_word = &p.rs_state->tile_epoch[blockIdx.x * kRsMaxTokenTiles + blockIdx.y];
      const uint32_t epoch = epoch_pre + 1u;
      // The fp32 tile goes through shared memory (behind the split-K landing zone of the idle pipeline stages) so
      // that the push works on token rows: a quarter row (32 columns) per thread, 16-byte accesses, long
      // contiguous runs per token towards the owner.
      constexpr int kRowPad = kTileN + 4;   // floats per row: shifts consecutive rows by four banks
      float* tile_s = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw))) + (S - 1) * TN * 128;
      if (pushes) {
        for (int c = 0; c < TN; c += kChunk) {
          if (t0 + c >= p.T) break;
          float v[kChunk];
          load_acc(c, v);
#pragma unroll
          for (int j = 0; j < kChunk; ++j) tile_s[(c + j) * kRowPad + warp * 32 + lane] = v[j];
        }
      }
      if (threadIdx.x == 0) rs_ok = 1;
      __syncthreads();
      if (pushes) {
        // hop 1: rows of the tile into the owner's receive buffer [src][T_cap][slice] of (value, epoch) pairs --
        // the owner's own tiles take the same road (into its own buffer), so that the reduction below reads every
        // contribution the same way and can run on any CTA
        const int col = (threadIdx.x & 3) * 32;
        const int n_local = n0 + col - owner * p.slice_cols;
        uint2* dst = p.peer_recv_ll[owner] + static_cast<long long>(p.rank) * p.T_cap * p.slice_cols + n_local;
        for (int r = threadIdx.x >> 2; r < TN; r += 32) {
          const int t = t0 + r;
          if (t >= p.T) continue;
          const float4* src4 = reinterpret_cast<const float4*>(tile_s + r * kRowPad + col);
          uint4* dst4 = reinterpret_cast<uint4*>(dst + static_cast<long long>(t) * p.slice_cols);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 f = src4[q];
            dst4[2 * q] = make_uint4(__float_as_uint(f.x), epoch, __float_as_uint(f.y), epoch);
            dst4[2 * q + 1] = make_uint4(__float_as_uint(f.z), epoch, __float_as_uint(f.w), epoch);
          }
        }
        stamp(7);
      }
      // hop 2, spread over the grid: this rank owns T x slice_cols values; they are cut into units of one token x
      // eight columns, one unit per thread, and dealt to the leading CTAs of the grid.  A thread has the 64 bytes
      // of all `world` contributions in flight at once, so a unit costs one round of polling instead of one per
      // contribution (a tile's owner CTA reducing its whole tile alone needed 2 x (world - 1) dependent rounds).
      const int n_ctas = gridDim.x * gridDim.y;                       // (split-K helpers never get here)
      const int cta = blockIdx.x + gridDim.x * blockIdx.y;
      const int groups = p.slice_cols / 8;                            // 8-column groups per token
      const int units = p.T * groups;
      const int n_red = min(n_ctas, (units + 127) / 128);
      if (reduces && cta < n_red) {
        stamp(8);
        __nv_bfloat16* my_x = p.peer_x[p.rank];
        const uint2* recv = p.peer_recv_ll[p.rank];
        for (int u0 = cta * 128; u0 < units; u0 += n_red * 128) {    // uniform trip count per CTA
          const int u = u0 + threadIdx.x;
          const bool live0 = u < units;
          const int t = live0 ? u / groups : 0;
          const int cg = live0 ? u % groups : 0;
          const int n_first = p.rank * p.slice_cols + cg * 8;         // first output column of the unit
          bool live = live0;
          float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          uint4 rv = make_uint4(0, 0, 0, 0);
          if (live) {
            rv = *reinterpret_cast<const uint4*>(my_x + static_cast<long long>(t) * p.ld_resid + n_first);
            uint4 v[kMaxRanks][4];
            bool here = false;
            for (uint32_t spin = 0; spin < kPeerPollLimit && !here; ++spin) {
              here = true;
#pragma unroll
              for (int src = 0; src < kMaxRanks; ++src) {
                if (src >= p.world) break;
                const uint4* sp = reinterpret_cast<const uint4*>(recv + (static_cast<long long>(src) * p.T_cap + t) * p.slice_cols + cg * 8);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  v[src][q] = ld_volatile_v4(sp + q);
                  here = here && v[src][q].y == epoch && v[src][q].w == epoch;
                }
              }
              if (!here) {
                if ((spin & 1023u) == 1023u && p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) break;
                if (spin > 64) __nanosleep(100);
              }
            }
            if (!here) {   // bounded: record it and let the step fail on the host instead of hanging
              report_status(p.status, kStatusPeerWaitTimeout);
              rs_ok = 0;
              live = false;
            }
#pragma unroll
            for (int src = 0; src < kMaxRanks; ++src) {   // rank order, the same on every rank
              if (src >= p.world) break;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                a[2 * q] += __uint_as_float(v[src][q].x);
                a[2 * q + 1] += __uint_as_float(v[src][q].z);
              }
            }
          }
          float ss = 0.f;
          if (live) {
            const __nv_bfloat162* rp = reinterpret_cast<const __nv_bfloat162*>(&rv);
            uint4 o;
            uint32_t* op = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              op[e] = pack_bf16x2(a[2 * e] + __bfloat162float(rp[e].x), a[2 * e + 1] + __bfloat162float(rp[e].y));
              const __nv_bfloat162 ob = *reinterpret_cast<const __nv_bfloat162*>(&op[e]);
              const float f0 = __bfloat162float(ob.x), f1 = __bfloat162float(ob.y);
              ss += f0 * f0 + f1 * f1;
            }
            const long long at = static_cast<long long>(t) * p.ld_resid + n_first;
            for (int rk = 0; rk < p.world; ++rk)   // all-gather by push (own copy included)
              *reinterpret_cast<uint4*>(p.peer_x[rk] + at) = o;
          }
          // the sixteen threads of one (token, 128-column tile): its sum of squares (a dead unit adds zero)
#pragma unroll
          for (int o2 = 1; o2 < 16; o2 <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o2);
          if (live && (threadIdx.x & 15) == 0) {
            const int tile_global = n_first / kTileN;
            for (int rk = 0; rk < p.world; ++rk)
              p.peer_ss[rk][static_cast<long long>(t) * kRsSsStride + tile_global] = ss;
          }
        }
        stamp(9);
        __syncthreads();
        stamp(10);
        // the block barrier orders every thread's peer stores before the signalling threads, whose release (system
        // scope) is cumulative over them: no separate fence
        if (rs_ok && threadIdx.x < p.world) red_release_sys_add(p.peer_xflag[threadIdx.x], 1u);
        stamp(11);
      }
      if (threadIdx.x == 0 && p.rs_phase != 1) *epoch_word = epoch;
      // what the next consumer of the residual stream has to wait for: one arrival per reducing CTA of every rank
      if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && p.rs_phase != 1)
        p.rs_state->x_expected += static_cast<unsigned int>(n_red * p.world);
    } else {
      const int n = n0 + warp * 32 + lane;
      const float bias = ((EPI == kEpiStore || EPI == kEpiResidual) && p.bias != nullptr && n < p.N) ? p.bias[n] : 0.f;
      const float act_a = EPI == kEpiStore && p.act_params != nullptr ? p.act_params[0] : 0.f;
      const float act_b = EPI == kEpiStore && p.act_params != nullptr ? p.act_params[1] : 0.f;
      // tiles of conv channels (kEpiStore at decode): taps + SiLU + history roll here, activation to conv_out
      const bool conv_tile = EPI == kEpiStore && p.conv_state != nullptr && n0 < p.conv_C;
      float cw[4] = {0.f, 0.f, 0.f, 0.f};
      if (conv_tile) {
        const uint2 wv = *reinterpret_cast<const uint2*>(p.conv_w + static_cast<long long>(n) * 4);
        const __nv_bfloat16* wp = reinterpret_cast<const __nv_bfloat16*>(&wv);
#pragma unroll
        for (int j = 0; j < 4; ++j) cw[j] = __bfloat162float(wp[j]);
      }
      __nv_bfloat16* const outp = conv_tile ? p.conv_out : p.out;
      const long long ldo = conv_tile ? p.conv_C : p.ldo;
      for (int c = 0; c < TN; c += kChunk) {
        if (t0 + c >= p.T) break;
        float v[kChunk];
        load_acc(c, v);
        if (conv_tile) {
          // all history columns of the chunk's tokens first (48 independent loads), then taps and the roll
          long long at[kChunk];
          __nv_bfloat16 h[kChunk][3];
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            const int t = t0 + c + j;
            at[j] = t < p.T ? static_cast<long long>(p.conv_slot[t]) * 3 * p.conv_C + n : -1;
          }
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            if (at[j] >= 0) {
              h[j][0] = p.conv_state[at[j]];
              h[j][1] = p.conv_state[at[j] + p.conv_C];
              h[j][2] = p.conv_state[at[j] + 2 * p.conv_C];
            }
          }
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            if (at[j] >= 0) {
              const __nv_bfloat16 xb = __float2bfloat16(v[j] + bias);   // the projection's bf16 value
              float a = 0.f;
              a += cw[0] * __bfloat162float(h[j][0]);
              a += cw[1] * __bfloat162float(h[j][1]);
              a += cw[2] * __bfloat162float(h[j][2]);
              a += cw[3] * __bfloat162float(xb);
              p.conv_state[at[j]] = h[j][1];
              p.conv_state[at[j] + p.conv_C] = h[j][2];
              p.conv_state[at[j] + 2 * p.conv_C] = xb;
              v[j] = a / (1.f + __expf(-a)) - bias;   // (the bias is added back below; it is zero for these tiles)
            }
          }
        }
        if constexpr (EPI == kEpiPartial) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            const int t = t0 + c + j;
            if (t < p.T && n < p.N)
              p.partial[(static_cast<long long>(blockIdx.z) * p.T + t) * p.N + n] = v[j];
          }
        } else if constexpr (EPI == kEpiPushAll) {
          // one-shot all-reduce by push: the fp32 tile goes to EVERY rank's receive buffer
          // [parity][src_rank][T_cap][N]; the reader sums the W sources in rank order.
          const unsigned int par = *p.call_idx & 1u;
          const long long base = ((static_cast<long long>(par) * p.world + p.rank) * p.T_cap) * p.N + n;
          for (int r = 0; r < p.world; ++r) {
            float* dst = p.peer_recv[r] + base;
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
              const int t = t0 + c + j;
              if (t < p.T && n < p.N) dst[static_cast<long long>(t) * p.N] = v[j];
            }
          }
        } else {
          // The residual may alias the output (in-place update): fetch the whole chunk's residual values
          // before the first store, otherwise every load would have to wait for the previous store.
          __nv_bfloat162 r2[kChunk / 2];
          if constexpr (EPI == kEpiResidual) {
#pragma unroll
            for (int m = 0; m < kChunk / 2; ++m) {
              const int t = t0 + c + 2 * m + (lane & 1);
              const int ne = n & ~1;
              r2[m] = (t < p.T && ne < p.N)
                          ? *reinterpret_cast<const __nv_bfloat162*>(p.resid + static_cast<long long>(t) * p.ldr + ne)
                          : __nv_bfloat162();
            }
          }
#pragma unroll
          for (int m = 0; m < kChunk / 2; ++m) {
            float a0 = v[2 * m] + bias;
            float a1 = v[2 * m + 1] + bias;
            if constexpr (EPI == kEpiStore) {
              if (p.act != kActNone) {
                a0 = activate(a0, p.act, act_a, act_b);
                a1 = activate(a1, p.act, act_a, act_b);
              }
            }
            const float send = (lane & 1) ? a0 : a1;
            const float recv = __shfl_xor_sync(0xffffffffu, send, 1);
            const int t = t0 + c + 2 * m + (lane & 1);
            const int ne = n & ~1;
            if (t < p.T && ne < p.N) {
              float lo = (lane & 1) ? recv : a0;
              float hi = (lane & 1) ? a1 : recv;
              if constexpr (EPI == kEpiResidual) {
                lo += __bfloat162float(r2[m].x);
                hi += __bfloat162float(r2[m].y);
              }
              if (EPI == kEpiStore && p.out32 != nullptr && ne >= p.out32_from)
                *reinterpret_cast<float2*>(p.out32 + static_cast<long long>(t) * p.ldo32 + ne - p.out32_from) = make_float2(lo, hi);
              else
                *reinterpret_cast<uint32_t*>(outp + static_cast<long long>(t) * ldo + ne) = pack_bf16x2(lo, hi);
            }
          }
        }
      }
      if constexpr (EPI == kEpiPushAll) {
        __syncthreads();
        if (threadIdx.x < p.world) {
          __threadfence_system();
          unsigned int* flag = p.peer_flag[threadIdx.x];
          asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(flag) : "memory");
        }
      }
    }
  }

  stamp(5);
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem_base, Cfg::kTmemCols);
  stamp(6);
}

// ------------------------------------------------------------------------------------------------------------
// Persistent kernel for more than 32 tokens, and for SwiGLU of up to 32 whose weight tiles fill whole rounds.  A walker, one
// CTA or a pair of CTAs (a cluster of two), goes over output tiles of 128 weight rows a CTA x `tn` tokens, with the roles split
// over ten warps so that the epilogue of tile i overlaps the main loop of tile i + 1:
//   warp 0  TMA producer (as many stages as fit, one running counter over tiles)
//   warp 1  MMA issuer; the fp32 accumulator alternates between TMEM columns [0, 256) and [256, 512)
//   warps 2..9  epilogue: warp w drains TMEM lanes 32 (w % 4) .., every second chunk of 16 tokens; tcgen05.ld -> bias /
//               activation / residual / SwiGLU -> bf16
// Two warps per lane group, because with short contractions (K = 2048: 13 us per 128 x 256 tile) one warp per group took
// longer to drain a tile than the tensor core to fill the next.  Tiles are numbered token-tile fastest, so the CTAs
// running at one time share a few weight tiles and all token tiles through L2.
//
// A single CTA is bound by its shared memory: a k-block of 128 x 64 weights and 256 x 64 tokens is 48 KB written by TMA and
// 48 KB read by the tensor core at 128 bytes a clock, 390 ns, where the products take 260.  A pair shares the tokens: each CTA
// loads its own weight rows and half of the tile's tokens (32 KB a k-block, seven stages instead of four), and the even CTA's
// instruction multiplies 256 weight rows by all tokens.  That is less traffic from L2 as well, and under the power cap less
// traffic is more clock.  Both forms give the same bits.  Back to back, weights from HBM, us, one CTA a tile -> pair: 2048 tokens
// 34816 x 5120 SwiGLU 488 -> 463, 5120 x 17408 residual 283 -> 251, 5120 x 6144 97 -> 89, 12352 x 2048 82 -> 75, 8192 x 2048
// 55 -> 51; 300 tokens 34816 x 5120 107 -> 99, 5120 x 17408 70 -> 63; for seconds at the power cap 34816 x 5120 573 -> 543,
// 14336 x 5120 262 -> 226.
constexpr int kPersistMaxTN = 256;
constexpr int kPersistMinTN = 64;   // narrowest single-CTA tile that pick_persist weighs (SwiGLU of up to 32 tokens: 16 or 32)
constexpr int kPairMinTN = 32;      // narrowest tile of a pair
constexpr int kPersistMaxStages = 12;
constexpr int kPersistEpiWarps = 8;
constexpr int kPersistThreads = 64 + 32 * kPersistEpiWarps;
constexpr int kPersistSmemBytes = 226 * 1024;
constexpr int kPersistExchangeBytes = 4 * 2 * 2 * 8 * 32 * 4;   // SwiGLU: per warp pair two buffers x two directions x 8 x 32
constexpr int persist_ring_bytes(int epi) { return kPersistSmemBytes - 1024 - (epi == kEpiSwiglu ? kPersistExchangeBytes : 0); }
// Time of one k-block of 64 by tokens per tile, all SMs busy, through widths of 64 (one CTA) or 32 (pair) to 256 tokens on
// weights of 5120 x 17408 and 34816 x 5120.  One CTA: 245 ns at 64, 311 at 128, 350 at 192, 400 at 256; where only four stages
// fit, from 240 tokens or, beside SwiGLU's exchange, from 208, another 20 ns.  Pair: 192 ns at 32, 218 at 64, 265 at 128 and
// 160 (weights from L2), then by the products: 300 at 192, 374 at 256.
constexpr double persist_kblock_ns(int tn, int epi) {
  return 215. + 0.65 * tn + (persist_ring_bytes(epi) / (kWTileBytes + 128 * tn) < 5 ? 20. : 0.);
}
constexpr double pair_kblock_ns(int tn) {
  return tn >= 160 ? 264. + 1.18 * (tn - 160) : tn >= 128 ? 264. : 264. - 0.81 * (128 - tn);
}
constexpr double kPairStartNs = 1500.;    // cluster launch, its barriers and the farther commit
// Per token of the last tile, whose epilogue nothing overlaps.  (The epilogue alone takes 14 now.  That, or 20, is the better with
// contractions up to K = 512, and for 12288 x 1024, 129 tokens, 10.0 us for 13.1; but 16480 x 5120, 1466 tokens, then takes wider
// tiles in fewer rounds, 206 for 184, and 24576 x 4096, 1884 tokens, 296 for 274.)
constexpr double kPersistTailNs = 30.;

template <int EPI, bool PAIR>
__global__ void __launch_bounds__(kPersistThreads, 1) gemm_persist_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                                           const __grid_constant__ CUtensorMap tmap_x,
                                                                           const KernelParams p) {
  static_assert(EPI == kEpiStore || EPI == kEpiResidual || EPI == kEpiSwiglu, "persistent kernel: plain epilogues only");
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kPersistMaxStages];
  __shared__ __align__(8) uint64_t bar_empty[kPersistMaxStages];
  __shared__ __align__(8) uint64_t bar_acc_full[2];
  __shared__ __align__(8) uint64_t bar_acc_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int TN = p.tn;
  // PAIR: the two CTAs of a cluster work on one tile of twice the weight rows; each loads its own rows and half of the tokens
  const int crank = PAIR ? static_cast<int>(blockIdx.x & 1) : 0;
  const int walker = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int walkers = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  const int x_rows = PAIR ? TN / 2 : TN;
  const int stage_bytes = kWTileBytes + x_rows * 128;
  constexpr int kRingBytes = persist_ring_bytes(EPI);
  const int n_stages = min(kPersistMaxStages, kRingBytes / stage_bytes);
  const int w_rows = (EPI == kEpiSwiglu) ? 64 : kTileN;                 // output rows per CTA and tile
  const int tile_rows = PAIR ? 2 * w_rows : w_rows;
  const int n_w_tiles = ((EPI == kEpiSwiglu ? p.swiglu_half : p.N) + tile_rows - 1) / tile_rows;
  const int n_t_tiles = (p.T + TN - 1) / TN;
  const int n_tiles = n_w_tiles * n_t_tiles;
  const int num_kb = p.num_kb;
  volatile int* abortp = &abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < n_stages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_acc_full[a]), 1);
      mbar_init(smem_u32(&bar_acc_empty[a]), PAIR ? 2 * kPersistEpiWarps : kPersistEpiWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
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

  if (warp == 0) {
    if (elect_one()) {
      // ---------------- TMA producer ----------------
      const uint64_t pol_w = l2_policy_evict_first();
      const uint64_t pol_x = l2_policy_evict_last();
      int s = 0;
      uint32_t ph = 1;      // the first pass over the ring finds every stage free
      uint32_t issued = 0;
      // (a pair's stage is counted by the even CTA's barrier, for both halves)
      auto load = [&](uint32_t dst, const CUtensorMap* map, int kb, int row, uint64_t pol) {
        const uint32_t full = smem_u32(&bar_full[s]);
        if constexpr (PAIR) tma_load_2d_pair(dst, map, mapa_shared(full, 0), kb * kBlockK, row, pol);
        else tma_load_2d(dst, map, full, kb * kBlockK, row, pol);
      };
      auto load_w = [&](int n0, int kb) {
        const uint32_t dst = smem_base + s * stage_bytes;
        if (crank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), PAIR ? 2 * stage_bytes : stage_bytes);
        load(dst, &tmap_w, kb, n0, pol_w);
        load(dst + 64 * 128, &tmap_w, kb, (EPI == kEpiSwiglu) ? p.swiglu_half + n0 : n0 + 64, pol_w);
      };
      auto load_x = [&](int t0, int kb) { load(smem_base + s * stage_bytes + kWTileBytes, &tmap_x, kb, t0, pol_x); };
      // Weights do not depend on the previous kernel: the ring is filled with them before it is waited for.
      const int primed = min(n_stages, num_kb);
      {
        const int n0 = walker / n_t_tiles * tile_rows + crank * w_rows, t0 = walker % n_t_tiles * TN + crank * x_rows;
        for (s = 0; s < primed; ++s) load_w(n0, s);
        pdl_wait_prior();  // activations are produced by the previous kernel
        for (s = 0; s < primed; ++s) load_x(t0, s);
        issued = static_cast<uint32_t>(primed);
        if (s == n_stages) { s = 0; ph ^= 1; }
      }
      int kb0 = primed;
      for (int tile = walker; tile < n_tiles && !*abortp; tile += walkers) {
        const int n0 = (tile / n_t_tiles) * tile_rows + crank * w_rows;
        const int t0 = (tile % n_t_tiles) * TN + crank * x_rows;
        bool ok = true;
        for (int kb = kb0; kb < num_kb; ++kb, ++issued) {
          if (!mbar_wait(smem_u32(&bar_empty[s]), ph, &abort_flag, p.status, kStatusEmptyWaitTimeout)) {
            ok = false;
            break;
          }
          load_w(n0, kb);
          load_x(t0, kb);
          if (++s == n_stages) { s = 0; ph ^= 1; }
        }
        kb0 = 0;
        if (!ok) break;
      }
      if (!*abortp && p.pf_per_cta > 0) {
        // own loads are all in flight: pull this CTA's share of the next kernel's weights into L2
        const long long off = static_cast<long long>(blockIdx.x) * p.pf_per_cta;
        if (off < p.pf_bytes) {
          const long long n = min(static_cast<long long>(p.pf_per_cta), p.pf_bytes - off) & ~15LL;
          if (n > 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.pf_ptr + off), "r"(static_cast<uint32_t>(n)) : "memory");
        }
      }
      if (*abortp) {
        // Unwinding: let copies that were already issued land before the CTA exits.  (The odd CTA of a pair has no barrier to
        // see them by: its own never completes, and the polls are the pause.)
        const uint32_t depth = static_cast<uint32_t>(n_stages);
        for (uint32_t j = issued > depth ? issued - depth : 0; j < issued; ++j) {
          const uint32_t bar = smem_u32(&bar_full[j % depth]);
          for (uint32_t spin = 0; spin < (1u << 20); ++spin)
            if (mbar_try_wait(bar, (j / depth) & 1)) break;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (crank == 0 && elect_one()) {
      // ---------------- MMA issuer (of both CTAs of a pair) ----------------
      const uint32_t idesc = umma_idesc(PAIR ? 2 * kTileN : kTileN, TN, 1, 1);
      int s = 0;
      uint32_t ph = 0;
      int tile_i = 0;
      auto commit = [](uint32_t bar) {
        if constexpr (PAIR) tc_commit_pair(bar);
        else tc_commit(bar);
      };
      for (int tile = walker; tile < n_tiles && !*abortp; tile += walkers, ++tile_i) {
        const int a = tile_i & 1;
        const uint32_t aph = (tile_i >> 1) & 1;
        // the epilogue has drained this accumulator's previous tile
        if (tile_i >= 2 &&
            !mbar_wait(smem_u32(&bar_acc_empty[a]), aph ^ 1, &abort_flag, p.status, kStatusAccumWaitTimeout))
          break;
        tc_fence_after();
        const uint32_t acc = tmem_base + a * kPersistMaxTN;
        bool ok = true;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&bar_full[s]), ph, &abort_flag, p.status, kStatusTmaWaitTimeout)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_base + s * stage_bytes;
          const uint64_t a_desc = umma_desc_k_sw128(a_addr);
          const uint64_t b_desc = umma_desc_k_sw128(a_addr + kWTileBytes);
#pragma unroll
          for (int k = 0; k < kBlockK / 16; ++k) {
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
    pdl_wait_prior();   // the residual may be written by the previous kernel
    const int lg = warp & 3;          // TMEM lane group this warp may read
    const int half = (warp - 2) >> 2; // which chunks: half, half + 2, ...
    constexpr int kChunk = 16;
    float* const xch_s = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)) + kRingBytes);
    const int pair = (lg & 1) + 2 * half;
    const uint32_t select = swap_select(lane);
    int tile_i = 0, xch_i = 0;
    for (int tile = walker; tile < n_tiles; tile += walkers, ++tile_i) {
      const int a = tile_i & 1;
      const uint32_t ph = (tile_i >> 1) & 1;
      const bool have = mbar_wait(smem_u32(&bar_acc_full[a]), ph, &abort_flag, p.status, kStatusAccumWaitTimeout);
      // one verdict for the eight warps, so that the pair barriers below are never divergent
      if (!epi_all(have && !*abortp)) break;
      tc_fence_after();
      const int n0 = (tile / n_t_tiles) * tile_rows + crank * w_rows;
      const int t0 = (tile % n_t_tiles) * TN;
      const int cols = min(TN, p.T - t0);     // live tokens of the tile
      const uint32_t lane_taddr = tmem_base + a * kPersistMaxTN + (static_cast<uint32_t>(lg * 32) << 16);
      if constexpr (EPI == kEpiSwiglu) {
        // Lane groups 0, 1 hold gate rows, 2, 3 the matching up rows.  The two warps of a pair swap eight of a chunk's
        // sixteen columns, so that both finish half of the units.
        const bool is_up = lg >= 2;
        const int n = n0 + (lg & 1) * 32 + lane;
        const int ne = n & ~1;
        for (int c = half * kChunk; c < cols; c += 2 * kChunk, ++xch_i) {
          float* buf = xch_s + (pair * 2 + (xch_i & 1)) * (2 * 8 * 32);
          float* mine = buf + (is_up ? 8 * 32 : 0);
          const float* other = buf + (is_up ? 0 : 8 * 32);
          uint32_t v[kChunk];
          tmem_ld_x16(lane_taddr + c, v);
          tmem_ld_wait_x16(v);
          // (selects, not indices: the chunk stays in registers)
#pragma unroll
          for (int j = 0; j < 8; ++j) mine[j * 32 + lane] = __uint_as_float(is_up ? v[j] : v[8 + j]);
          epi_pair_sync(pair);
          const int tb = t0 + c + (is_up ? 8 : 0);
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
          const int live = ne < p.swiglu_half ? (p.T - tb - (lane & 1) + 1) >> 1 : 0;
          store_rows<4>({p.out + static_cast<long long>(tb + (lane & 1)) * p.ldo + ne, 2 * p.ldo, live}, w);
        }
      } else {
        const int n = n0 + lg * 32 + lane;
        const int ne = n & ~1;
        const float bias = (p.bias != nullptr && n < p.N) ? p.bias[n] : 0.f;
        const float act_a = EPI == kEpiStore && p.act_params != nullptr ? p.act_params[0] : 0.f;
        const float act_b = EPI == kEpiStore && p.act_params != nullptr ? p.act_params[1] : 0.f;
        const bool has32 = EPI == kEpiStore && p.out32 != nullptr && n0 + kTileN > p.out32_from;   // (of the tile)
        const bool all32 = has32 && n0 >= p.out32_from;
        const long long row0 = t0 + (lane & 1);
        auto live = [&](int c) { return ne < p.N ? min(8, (p.T - t0 - c - (lane & 1) + 1) >> 1) : 0; };
        // The residual may alias the output (in-place update): a chunk's values are fetched one chunk ahead, so that
        // their latency runs beside the chunk before and no load waits for a store.
        uint32_t r2[kChunk / 2];
        auto fetch = [&](int c) { load_rows8({p.resid + (row0 + c) * p.ldr + ne, 2 * p.ldr, live(c)}, r2); };
        if constexpr (EPI == kEpiResidual) fetch(half * kChunk);
        for (int c = half * kChunk; c < cols; c += 2 * kChunk) {
          uint32_t r[kChunk / 2];
          if constexpr (EPI == kEpiResidual) {
#pragma unroll
            for (int m = 0; m < kChunk / 2; ++m) r[m] = r2[m];
            if (c + 2 * kChunk < cols) fetch(c + 2 * kChunk);
          }
          uint32_t v[kChunk];
          tmem_ld_x16(lane_taddr + c, v);
          tmem_ld_wait_x16(v);
          float f[kChunk];
#pragma unroll
          for (int j = 0; j < kChunk; ++j) f[j] = __uint_as_float(v[j]) + bias;
          if constexpr (EPI == kEpiStore) {
            if (p.act == kActXielu) {
#pragma unroll
              for (int j = 0; j < kChunk; ++j) f[j] = activate(f[j], kActXielu, act_a, act_b);
            } else if (p.act != kActNone) {
#pragma unroll
              for (int j = 0; j < kChunk; ++j) f[j] = activate(f[j], p.act, act_a, act_b);
            }
          }
          if (!has32) {
            store_chunk<EPI == kEpiResidual>({p.out + (row0 + c) * p.ldo + ne, 2 * p.ldo, live(c)}, f, r, select);
          } else if (all32) {
            // fp32 columns: a warp's 32 of a token are a line of 128 bytes as they are
            float* at = p.out32 + (t0 + c) * static_cast<long long>(p.ldo32) + n - p.out32_from;
            const int n_live = n < p.N ? p.T - t0 - c : 0;
            if (n_live >= kChunk) {
#pragma unroll
              for (int j = 0; j < kChunk; ++j, at += p.ldo32) *at = f[j];
            } else {
#pragma unroll
              for (int j = 0; j < kChunk; ++j, at += p.ldo32)
                if (j < n_live) *at = f[j];
            }
          } else {
            // columns from out32_from on as fp32, those before as bf16: pairs swapped in full
            const int n_live = live(c);
#pragma unroll
            for (int m = 0; m < kChunk / 2; ++m) {
              const float recv = __shfl_xor_sync(0xffffffffu, (lane & 1) ? f[2 * m] : f[2 * m + 1], 1);
              const float lo = (lane & 1) ? recv : f[2 * m], hi = (lane & 1) ? f[2 * m + 1] : recv;
              const long long t = row0 + c + 2 * m;
              if (m < n_live) {
                if (ne >= p.out32_from) *reinterpret_cast<float2*>(p.out32 + t * p.ldo32 + ne - p.out32_from) = make_float2(lo, hi);
                else *reinterpret_cast<uint32_t*>(p.out + t * p.ldo + ne) = pack_bf16x2(lo, hi);
              }
            }
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

// Tokens per tile of the persistent kernel and whether pairs of CTAs walk them: the width (a multiple of 16) and form with the
// least estimated time.  `rows` output rows in tiles of 128 a CTA (64 beside SwiGLU) times the token tiles are dealt out in
// rounds of one tile per walker; what a fixed 256 loses is the last round (N = 5120, T = 2048: 160 tiles of 74 pairs = 2.16
// rounds, paid as 3; 192 tokens make it 2.97) or, with few tiles, the SMs that get none (N = 264: 16 tiles of 256 tokens
// against 64 of 64).  One CTA a tile is left with short contractions (us, one CTA and pair: 2048 tokens 2048 x 512 9.3 and
// 10.7, 2048 x 2048 16.9 and 17.9; 64 tokens 34816 x 128 6.1 and 9.2, 8.7 before there were pairs; 96 tokens 12288 x 512 7.6 and
// 9.0; 128 tokens 12288 x 1024 10.1 and 13.1); from K = 2048 on pairs were the faster at every size tried up to 128 tokens.
struct PersistPlan { int tn; bool pair; };
PersistPlan pick_persist(int T, int rows, int num_kb, int sms, int epi) {
  PersistPlan best = {kPersistMaxTN, true};
  double best_ns = 0;
  const int cta_rows = epi == kEpiSwiglu ? 64 : kTileN;
  for (int pair = 1; pair >= 0; --pair) {
    const int w_tiles = (rows + (cta_rows << pair) - 1) / (cta_rows << pair);
    for (int tn = kPersistMaxTN; tn >= (pair ? kPairMinTN : kPersistMinTN); tn -= 16) {
      const long long tiles = static_cast<long long>(w_tiles) * ((T + tn - 1) / tn);
      const long long rounds = (tiles + (sms >> pair) - 1) / (sms >> pair);
      const double ns = static_cast<double>(rounds) * num_kb * (pair ? pair_kblock_ns(tn) : persist_kblock_ns(tn, epi)) +
                        kPersistTailNs * tn + (pair ? kPairStartNs : 0.);
      if (best_ns == 0 || ns < best_ns * 0.99) { best = {tn, pair != 0}; best_ns = ns; }
    }
  }
  return best;
}

template <int EPI, bool PAIR>
cudaError_t launch_walkers(const CUtensorMap& tw, const CUtensorMap& tx, const KernelParams& kp, int n_tiles,
                           cudaStream_t stream, bool pdl) {
  auto kern = gemm_persist_kernel<EPI, PAIR>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPersistSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  constexpr int kCtas = PAIR ? 2 : 1;
  const int walkers = device_sm_count() / kCtas;
  cfg.gridDim = dim3(kCtas * (n_tiles < walkers ? n_tiles : walkers));
  cfg.blockDim = dim3(kPersistThreads);
  cfg.dynamicSmemBytes = kPersistSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (PAIR) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = kCtas;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (pdl) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  return cudaLaunchKernelEx(&cfg, kern, tw, tx, kp);
}

template <int EPI>
cudaError_t launch_persist(bool pair, const CUtensorMap& tw, const CUtensorMap& tx, const KernelParams& kp, int n_tiles,
                           cudaStream_t stream, bool pdl) {
  return pair ? launch_walkers<EPI, true>(tw, tx, kp, n_tiles, stream, pdl) : launch_walkers<EPI, false>(tw, tx, kp, n_tiles, stream, pdl);
}

template <int TN, int EPI, bool DEEP>
cudaError_t launch_one(const CUtensorMap& tw, const CUtensorMap& tx, const KernelParams& kp, dim3 grid,
                       cudaStream_t stream, bool pdl) {
  using Cfg = GemmCfg<TN, DEEP>;
  auto kern = gemm_ws_kernel<TN, EPI, DEEP>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (kp.cluster > 1) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 1;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = kp.cluster;
    ++n_attr;
  }
  if (pdl) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  return cudaLaunchKernelEx(&cfg, kern, tw, tx, kp);
}

// One CTA per SM with the deep pipeline when the whole grid fits in one wave.  NFB_GEMM_DEEP=0 keeps the shallow
// pipeline (about 100 KB per CTA) for every size, so that the CTAs of two consecutive kernels fit on one SM and the
// next kernel's weight prefetch (programmatic dependent launch) can run under the current kernel.
bool deep_enabled() {
  static const bool enabled = [] {
    const char* e = getenv("NFB_GEMM_DEEP");
    return !(e != nullptr && e[0] == '0');
  }();
  return enabled;
}
bool use_deep(int tn, long long ctas) { return deep_enabled() && tn <= 64 && ctas <= device_sm_count(); }

template <int EPI>
cudaError_t launch_tn(int TN, const CUtensorMap& tw, const CUtensorMap& tx, const KernelParams& kp,
                      dim3 grid, cudaStream_t stream, bool pdl) {
  const bool deep = use_deep(TN, static_cast<long long>(grid.x) * grid.y * grid.z);
  switch (TN) {
    case 16: return deep ? launch_one<16, EPI, true>(tw, tx, kp, grid, stream, pdl)
                         : launch_one<16, EPI, false>(tw, tx, kp, grid, stream, pdl);
    case 32: return deep ? launch_one<32, EPI, true>(tw, tx, kp, grid, stream, pdl)
                         : launch_one<32, EPI, false>(tw, tx, kp, grid, stream, pdl);
    case 64: return deep ? launch_one<64, EPI, true>(tw, tx, kp, grid, stream, pdl)
                         : launch_one<64, EPI, false>(tw, tx, kp, grid, stream, pdl);
    case 128: return launch_one<128, EPI, false>(tw, tx, kp, grid, stream, pdl);
    default:
      return static_cast<long long>(grid.x) * grid.y * grid.z <= device_sm_count()
                 ? launch_one<256, EPI, true>(tw, tx, kp, grid, stream, pdl)
                 : launch_one<256, EPI, false>(tw, tx, kp, grid, stream, pdl);
  }
}

// Tensor maps are pure functions of (pointer, shape, box): cache them so the
// eager path does not re-encode on every call.
struct TmapKey {
  const void* base; uint64_t rows, cols, ld; uint32_t box_rows;
  bool operator==(const TmapKey& o) const {
    return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows;
  }
};
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.base);
    h = h * 1000003u ^ k.rows; h = h * 1000003u ^ k.cols; h = h * 1000003u ^ k.ld;
    return h * 1000003u ^ k.box_rows;
  }
};
bool cached_tmap(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows) {
  static std::mutex mu;
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  TmapKey key{base, rows, cols, ld, box_rows};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return true; }
  CUtensorMap m;
  if (!make_tmap_2d(&m, TmapDtype::BF16, base, rows, cols, ld, box_rows, kBlockK, true)) return false;
  if (cache.size() > 65536) cache.clear();
  cache.emplace(key, m);
  *out = m;
  return true;
}

}  // namespace

void gemm_trace_enable(bool on) { g_trace_enabled = on; }
void gemm_timeline_begin() {
  g_trace_enabled = true;
  g_timeline_next = 0;
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_gemm_timeline) == cudaSuccess) cudaMemset(p, 0, sizeof(unsigned long long) * kTimelineSlots * kTimelineCtas * kTraceStamps);
}
int gemm_timeline_end(unsigned long long* host, int* n_slots, int* n_ctas) {
  g_trace_enabled = false;
  const int used = g_timeline_next < 0 ? 0 : (g_timeline_next < kTimelineSlots ? g_timeline_next : kTimelineSlots);
  g_timeline_next = -1;
  *n_slots = kTimelineSlots;
  *n_ctas = kTimelineCtas;
  if (host != nullptr)
    cudaMemcpyFromSymbol(host, g_gemm_timeline, sizeof(unsigned long long) * kTimelineSlots * kTimelineCtas * kTraceStamps);
  return used;
}
int gemm_trace_read(unsigned long long* host, int n_ctas) {
  if (n_ctas > kTraceCtas) n_ctas = kTraceCtas;
  cudaMemcpyFromSymbol(host, g_gemm_trace, sizeof(unsigned long long) * n_ctas * kTraceStamps);
  return kTraceStamps;
}

int gemm_tile_tokens(int T) {
  if (T <= 16) return 16;
  if (T <= 32) return 32;
  if (T <= 64) return 64;
  if (T <= 128) return 128;
  return 256;
}

// Largest in-cluster split for a token tile: the leader needs (S-1) * TN * 512 bytes for the peers'
// fp32 tiles plus TN * 256 bytes for the SwiGLU exchange inside its idle pipeline stages.
int gemm_max_cluster(int tn) {
  switch (tn) {
    case 16: return 8;
    case 32: return 6;   // 5 stages x 20.5 KB hold 5 peer tiles of 16 KB plus the 8 KB SwiGLU exchange
    case 64: return 2;
    case 128: return 2;
    default: return 1;
  }
}

// How many clusters of `s` CTAs (along z) of one kernel instance can be resident at once.  A cluster lives inside
// one GPC, so this is not sm_count / s: with one CTA per SM, 17 clusters of 8 or 34 clusters of 4 do not fit and
// the grid runs in two waves.  Asked from the runtime once per (kernel, cluster size) and cached.
template <int TN, int EPI, bool DEEP>
int occupancy_clusters(int s) {
  using Cfg = GemmCfg<TN, DEEP>;
  auto kern = gemm_ws_kernel<TN, EPI, DEEP>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, 1, s);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = s;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

template <int EPI>
int occupancy_clusters_tn(int tn, bool deep, int s) {
  switch (tn) {
    case 16: return deep ? occupancy_clusters<16, EPI, true>(s) : occupancy_clusters<16, EPI, false>(s);
    case 32: return deep ? occupancy_clusters<32, EPI, true>(s) : occupancy_clusters<32, EPI, false>(s);
    case 64: return deep ? occupancy_clusters<64, EPI, true>(s) : occupancy_clusters<64, EPI, false>(s);
    default: return 0;
  }
}

// 0 = unknown (no device, query failed): the caller then falls back to the SM-count estimate.
int max_active_clusters(int tn, int epi, bool deep, int s) {
  static std::mutex mu;
  static std::unordered_map<int, int> cache;
  const int key = ((tn * 16 + epi) * 2 + (deep ? 1 : 0)) * 16 + s;
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  int n = 0;
  switch (epi) {
    case kEpiStore: n = occupancy_clusters_tn<kEpiStore>(tn, deep, s); break;
    case kEpiResidual: n = occupancy_clusters_tn<kEpiResidual>(tn, deep, s); break;
    case kEpiSwiglu: n = occupancy_clusters_tn<kEpiSwiglu>(tn, deep, s); break;
    case kEpiPushAll: n = occupancy_clusters_tn<kEpiPushAll>(tn, deep, s); break;
    case kEpiRsAg: n = occupancy_clusters_tn<kEpiRsAg>(tn, deep, s); break;
    default: n = 0;
  }
  cache.emplace(key, n);
  return n;
}

int gemm_pick_splits(int T, int N, int K, int epi, int sm_count) {
  const int tn = gemm_tile_tokens(T);
  const int rows = epi == kEpiSwiglu ? N / 2 : N;
  const int tile_rows = epi == kEpiSwiglu ? 64 : kTileN;
  const int tiles = ((rows + tile_rows - 1) / tile_rows) * ((T + tn - 1) / tn);
  const int num_kb = (K + kBlockK - 1) / kBlockK;
  const bool in_cluster = epi != kEpiPartial && epi != kEpiPushPartial;
  if (T > 256) return 1;
  if (!in_cluster) {
    const int slots = sm_count * (tn <= 64 ? 2 : 1);
    if (tiles >= slots) return 1;
    int s = slots / tiles;
    if (s > 8) s = 8;
    while (s > 1 && num_kb / s < 8) --s;
    const int per = (num_kb + s - 1) / s;
    return (num_kb + per - 1) / per;
  }
  // in-cluster split: aim for ONE wave of deep-pipeline CTAs (<= sm_count CTAs, one per SM)
  if (tiles >= sm_count || tn > 64) return 1;
  int s = sm_count / tiles;
  if (s > 8) s = 8;
  if (tn == 64 && s > 6) s = 6;
  if (tn == 64 && epi == kEpiRsAg && s > 5) s = 5;   // its row staging tile shares the pipeline stages
  if ((!deep_enabled() || epi == kEpiSwiglu) && s > gemm_max_cluster(tn)) s = gemm_max_cluster(tn);
  // the largest split whose clusters are all resident at once (one wave), that leaves every split at least eight
  // k-blocks and no split empty
  for (; s > 1; --s) {
    if (num_kb / s < 8) continue;
    if ((num_kb + s - 1) / s * (s - 1) >= num_kb) continue;
    const bool deep = use_deep(tn, static_cast<long long>(tiles) * s);
    if (!deep && s > gemm_max_cluster(tn)) continue;
    const int fit = max_active_clusters(tn, epi, deep, s);
    if (fit > 0 && fit < tiles) continue;
    break;
  }
  return s < 1 ? 1 : s;
}

const char* gemm_bf16(const GemmArgs& a) {
  if (a.T <= 0 || a.N <= 0 || a.K <= 0) return "gemm_bf16: empty problem";
  if ((a.K % 8) || (a.ldw % 8) || (a.ldx % 8)) return "gemm_bf16: K and leading dims must be multiples of 8";
  if ((reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.x)) & 15)
    return "gemm_bf16: operands must be 16-byte aligned";
  if ((a.N & 1) || (a.ldo & 1)) return "gemm_bf16: N and ldo must be even";
  if ((a.act == kActXielu || a.act == kActSoftcap) && a.act_params == nullptr) return "gemm_bf16: the activation needs its two parameters";
  if (a.out32 != nullptr) {
    if (a.epi != kEpiStore || a.conv.state != nullptr) return "gemm_bf16: fp32 columns need the plain store epilogue";
    if ((a.ldo32 & 1) || (a.out32_from & 1) || a.out32_from < 0 || a.out32_from >= a.N ||
        a.ldo32 < a.N - a.out32_from || (reinterpret_cast<uintptr_t>(a.out32) & 7))
      return "gemm_bf16: fp32 columns must start at an even column and have an even leading dimension";
  }
  const int tn = gemm_tile_tokens(static_cast<int>(a.T));
  const bool global_split = a.epi == kEpiPartial || a.epi == kEpiPushPartial;
  const bool plain = (a.epi == kEpiStore || a.epi == kEpiResidual || a.epi == kEpiSwiglu) && a.gather.flag == nullptr &&
                     a.conv.state == nullptr;
  KernelParams kp = {};
  kp.trace = g_trace_enabled ? 1 : 0;
  if (g_trace_enabled && g_timeline_next >= 0) kp.trace = 2 + (g_timeline_next++ % kTimelineSlots);
  kp.T = static_cast<int>(a.T); kp.N = static_cast<int>(a.N); kp.K = static_cast<int>(a.K);
  kp.num_kb = (kp.K + kBlockK - 1) / kBlockK;
  const int w_tiles = a.epi == kEpiSwiglu ? (kp.N / 2 + 63) / 64 : (kp.N + kTileN - 1) / kTileN;
  int splits = a.splits < 1 ? 1 : a.splits;
  if (splits > kp.num_kb) splits = kp.num_kb;
  if (splits != (a.splits < 1 ? 1 : a.splits)) return "gemm_bf16: split count leaves an empty split";
  kp.kb_per_split = (kp.num_kb + splits - 1) / splits;
  if ((kp.num_kb + kp.kb_per_split - 1) / kp.kb_per_split != splits) return "gemm_bf16: split count leaves an empty split";
  kp.cluster = 1;
  if (!global_split && splits > 1) {
    const long long ctas = static_cast<long long>((kp.N + kTileN - 1) / kTileN) * ((kp.T + tn - 1) / tn) * splits;
    const bool deep = use_deep(tn, ctas);  // (SwiGLU is checked against the shallow limit)
    const int cap = (deep && a.epi != kEpiSwiglu) ? (tn == 64 ? 6 : 8) : gemm_max_cluster(tn);
    if (splits > cap) return "gemm_bf16: in-cluster split exceeds the tile's limit";
    kp.cluster = splits;
  }
  if (a.epi == kEpiPushPartial || a.epi == kEpiPushAll || a.epi == kEpiRsAg) {
    if (a.world < 1 || a.world > kMaxRanks || a.rank < 0 || a.rank >= a.world) return "gemm_bf16: bad rank/world";
    kp.rank = a.rank;
    kp.world = a.world;
    for (int r = 0; r < a.world; ++r) {
      if (a.peer_recv[r] == nullptr || (a.peer_flag[r] == nullptr && a.epi != kEpiRsAg))
        return "gemm_bf16: missing peer pointer";
      kp.peer_recv[r] = a.peer_recv[r];
      kp.peer_flag[r] = a.peer_flag[r];
    }
  }
  if (a.epi == kEpiPushPartial) {
    if (kp.N % a.world || (kp.N / a.world) % kTileN) return "gemm_bf16: N / world must be a multiple of 128";
    kp.slice_cols = kp.N / a.world;
  }
  if (a.epi == kEpiPushAll) {
    if (a.call_idx == nullptr || a.T_cap < kp.T) return "gemm_bf16: push-all needs the call counter and T <= T_cap";
    kp.call_idx = a.call_idx;
    kp.T_cap = a.T_cap;
  }
  if (a.epi == kEpiRsAg) {
    if (kp.N % a.world || (kp.N / a.world) % kTileN) return "gemm_bf16: N / world must be a multiple of 128";
    if (kp.N / kTileN > kRsMaxTiles || kp.N / kTileN > kRsSsStride)
      return "gemm_bf16: too many column tiles for the reduce-scatter bookkeeping";
    if ((kp.T + tn - 1) / tn > kRsMaxTokenTiles || a.T_cap < kp.T) return "gemm_bf16: too many rows for the receive buffer";
    if (a.rs_state == nullptr || a.rs_phase < 0 || a.rs_phase > 2 || (a.ld_resid % 8))
      return "gemm_bf16: reduce-scatter epilogue needs its state, a phase in 0..2 and a residual stride that is a multiple of 8";
    if (kp.T > 128) return "gemm_bf16: reduce-scatter epilogue is for decode sizes (T <= 128)";
    // the fp32 tile is staged behind the split-K landing zone inside the pipeline stages
    if (tn == 64 && splits > 5) return "gemm_bf16: reduce-scatter epilogue with a 64-token tile allows at most 5 splits";
    for (int r = 0; r < a.world; ++r)
      if (reinterpret_cast<uintptr_t>(a.peer_x[r]) & 15) return "gemm_bf16: residual buffers must be 16-byte aligned";
    // an owner CTA waits for peers while it holds its SM: every CTA of the grid has to be resident at once
    if (a.rs_phase == 0 && static_cast<long long>(kp.N / kTileN) * ((kp.T + tn - 1) / tn) * splits > device_sm_count())
      return "gemm_bf16: reduce-scatter epilogue needs a grid that is resident at once";
    kp.slice_cols = kp.N / a.world;
    kp.T_cap = a.T_cap;
    kp.ld_resid = a.ld_resid;
    kp.rs_state = a.rs_state;
    kp.rs_phase = a.rs_phase;
    for (int r = 0; r < a.world; ++r) {
      if (a.peer_x[r] == nullptr || a.peer_ss[r] == nullptr || a.peer_xflag[r] == nullptr)
        return "gemm_bf16: missing residual pointer of a rank";
      kp.peer_x[r] = static_cast<__nv_bfloat16*>(a.peer_x[r]);
      kp.peer_recv_ll[r] = reinterpret_cast<uint2*>(a.peer_recv[r]);
      kp.peer_ss[r] = a.peer_ss[r];
      kp.peer_xflag[r] = a.peer_xflag[r];
    }
  }
  if (a.gather.flag != nullptr) {
    if (a.epi != kEpiStore && a.epi != kEpiSwiglu) return "gemm_bf16: the gathered input needs the store or SwiGLU epilogue";
    if (a.gather.target == nullptr || a.gather.ss == nullptr || a.gather.ss_tiles < 1 ||
        a.gather.ss_tiles > kRsSsStride || a.gather.n_features < 1 || kp.T > 256)
      return "gemm_bf16: bad gathered-input description";
    kp.g_flag = a.gather.flag;
    kp.g_target = a.gather.target;
    kp.g_ss = a.gather.ss;
    kp.g_tiles = a.gather.ss_tiles;
    kp.g_inv_n = 1.f / static_cast<float>(a.gather.n_features);
    kp.g_eps = a.gather.eps;
  }
  if (a.conv.state != nullptr) {
    if (a.epi != kEpiStore || a.bias != nullptr || a.act != kActNone)
      return "gemm_bf16: the conv epilogue needs the plain store epilogue";
    if (a.conv.w == nullptr || a.conv.slot == nullptr || a.conv.out == nullptr || a.conv.C <= 0 ||
        a.conv.C % kTileN || a.conv.C > kp.N || kp.T > 256)
      return "gemm_bf16: bad conv description (C must be a multiple of 128 within N, decode sizes only)";
    if (reinterpret_cast<uintptr_t>(a.conv.w) & 7) return "gemm_bf16: conv weights must be 8-byte aligned";
    kp.conv_w = static_cast<const __nv_bfloat16*>(a.conv.w);
    kp.conv_state = static_cast<__nv_bfloat16*>(a.conv.state);
    kp.conv_slot = a.conv.slot;
    kp.conv_out = static_cast<__nv_bfloat16*>(a.conv.out);
    kp.conv_C = a.conv.C;
  }
  kp.swiglu_half = a.epi == kEpiSwiglu ? kp.N / 2 : 0;
  kp.glu = a.glu;
  if (a.epi == kEpiSwiglu && (kp.N % 4)) return "gemm_bf16: SwiGLU needs N % 4 == 0";
  kp.out = static_cast<__nv_bfloat16*>(a.out); kp.ldo = a.ldo;
  kp.resid = static_cast<const __nv_bfloat16*>(a.resid); kp.ldr = a.ldr;
  kp.bias = a.bias; kp.act = a.epi == kEpiStore ? a.act : kActNone; kp.partial = a.partial; kp.status = a.status;
  if (a.epi == kEpiResidual && a.resid == nullptr) return "gemm_bf16: residual epilogue without residual";
  if (a.epi == kEpiPartial && a.partial == nullptr) return "gemm_bf16: split-K without workspace";
  kp.act_params = a.act_params; kp.out32 = a.out32; kp.ldo32 = a.ldo32; kp.out32_from = a.out32_from;
  const bool all32 = a.out32 != nullptr && a.out32_from == 0;
  const bool needs_out = !all32 && (a.epi == kEpiStore || a.epi == kEpiResidual || a.epi == kEpiSwiglu);
  if (needs_out && a.out == nullptr) return "gemm_bf16: no output";

  // More than 32 tokens and a plain epilogue: persistent kernel, epilogue overlapped with the next main loop.  One tile of 64,
  // 128 or 256 tokens per CTA, or narrower ones, before -> pairs now, us: 48 tokens 16480 x 5120 28.0 -> 26.9, 24576 x 4096
  // SwiGLU 42.0 -> 38.1; 80 tokens 34816 x 5120 SwiGLU 90 -> 54; 128 tokens 12352 x 2048 18.5 -> 14.0, 1024 x 2048 SwiGLU
  // 12.1 -> 9.6, 248320 x 2048 278 -> 166; 256 tokens 5120 x 17408 residual 67 -> 58.  Up to 32 tokens pairs lose what the
  // cluster costs (one token: 12352 x 2048 11.3 and 11.7, the language-model head 355 and 374) or, with a split contraction, more.
  // (NFB_GEMM_PERSISTENT=0 keeps the one-tile-per-CTA kernel for every size)
  static const bool persistent_enabled = [] {
    const char* e = getenv("NFB_GEMM_PERSISTENT");
    return !(e != nullptr && e[0] == '0');
  }();
  // Up to 32 tokens, SwiGLU with more weight tiles than SMs and at least three quarters of them busy in the last round: the
  // same kernel, one CTA a tile, streams the weights in whole rounds of one tile per SM, where two CTAs per SM run them in one.
  // 34816 x 5120, 272 tiles, 1.84 rounds: one token 70.1 -> 69.6 us; 24576 x 4096, 192 tiles, whose second round would
  // leave 104 SMs idle: one token 47.1 us with two CTAs per SM, 50.1 in rounds.  (The plain store gained nothing, the
  // language-model head lost 1 %.)
  const int last_round = w_tiles % device_sm_count();
  const bool stream = tn <= 32 && a.epi == kEpiSwiglu && w_tiles > device_sm_count() &&
                      (last_round == 0 || 4 * last_round >= 3 * device_sm_count());
  const bool persistent = (tn > 32 || stream) && splits == 1 && persistent_enabled && !g_trace_enabled && plain;
  const int out_rows = a.epi == kEpiSwiglu ? kp.N / 2 : kp.N;
  const PersistPlan plan = persistent && !stream ? pick_persist(kp.T, out_rows, kp.num_kb, device_sm_count(), a.epi) : PersistPlan{tn, false};
  kp.tn = plan.tn;

  CUtensorMap tw, tx;
  if (!cached_tmap(&tw, a.w, a.N, a.K, a.ldw, 64)) return "gemm_bf16: weight tensor map rejected";
  if (!cached_tmap(&tx, a.x, a.T, a.K, a.ldx, plan.pair ? plan.tn / 2 : plan.tn)) return "gemm_bf16: activation tensor map rejected";

  dim3 grid;
  grid.x = plan.pair ? (w_tiles + 1) / 2 : w_tiles;
  grid.y = (kp.T + plan.tn - 1) / plan.tn;
  grid.z = splits;
  if (a.prefetch != nullptr && a.prefetch_bytes > 0 && (reinterpret_cast<uintptr_t>(a.prefetch) & 15) == 0) {
    long long ctas = static_cast<long long>(grid.x) * grid.y * grid.z * (plan.pair ? 2 : 1);
    if (persistent && ctas > device_sm_count()) ctas = device_sm_count();
    long long per = (a.prefetch_bytes + ctas - 1) / ctas;
    per = (per + 4095) & ~4095LL;                 // whole 4 KB pieces per CTA
    if (per > (256 << 10)) per = 256 << 10;       // a quarter megabyte per CTA: a third of L2 when every SM asks
    kp.pf_ptr = static_cast<const uint8_t*>(a.prefetch);
    kp.pf_bytes = a.prefetch_bytes;
    kp.pf_per_cta = static_cast<int>(per);
  }
  cudaError_t e;
  if (persistent) {
    const int n_tiles = static_cast<int>(grid.x * grid.y);
    switch (a.epi) {
      case kEpiStore: e = launch_persist<kEpiStore>(plan.pair, tw, tx, kp, n_tiles, a.stream, a.pdl); break;
      case kEpiResidual: e = launch_persist<kEpiResidual>(plan.pair, tw, tx, kp, n_tiles, a.stream, a.pdl); break;
      default: e = launch_persist<kEpiSwiglu>(plan.pair, tw, tx, kp, n_tiles, a.stream, a.pdl); break;
    }
    return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
  }
  switch (a.epi) {
    case kEpiStore: e = launch_tn<kEpiStore>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    case kEpiResidual: e = launch_tn<kEpiResidual>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    case kEpiSwiglu: e = launch_tn<kEpiSwiglu>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    case kEpiPartial: e = launch_tn<kEpiPartial>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    case kEpiPushPartial: e = launch_tn<kEpiPushPartial>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    case kEpiPushAll: e = launch_tn<kEpiPushAll>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    case kEpiRsAg: e = launch_tn<kEpiRsAg>(tn, tw, tx, kp, grid, a.stream, a.pdl); break;
    default: return "gemm_bf16: unknown epilogue";
  }
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace nfb
