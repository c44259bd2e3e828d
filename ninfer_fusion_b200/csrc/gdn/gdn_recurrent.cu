// Gated delta-rule recurrence with the fp32 state held in registers for the
// whole token loop: one CTA per (value head, sequence).  Eight lanes share a
// state row (each owns 16 of its 128 columns as four interleaved float4), so a
// warp instruction moves four fully used 128-byte lines and a thread owns four
// rows -> 64 state registers, <= 128 registers in total, two CTAs per SM, which
// lets one CTA's state load overlap the other's store.  Fused in the same pass:
// q/k L2 normalisation, the gating non-linearities (softplus/exp/sigmoid) and the
// per-head gated RMSNorm epilogue, so a decode step reads and writes each 64 KB
// state exactly once.  Used for decode (1 token per sequence), verify
// (write_state = 0, state untouched, the accepted prefix is replayed afterwards
// with write_state = 1) and as the sequential prefill path.
//
// Reference: include/ninfer/ops/gated_delta_net.h:26-112, gdn_gating.h,
// gated_rmsnorm.h, src/ops/linear_attention/gated_delta_net/recurrent.cuh.
#include "gdn.h"

#include "../common/device.h"
#include "../common/ptx.cuh"
#include "../gemm/nvfp4_act.cuh"

namespace nfb {

namespace {

constexpr int kDk = 128, kDv = 128;
constexpr int kThreads = 256;
constexpr int kRowsPerThread = 4;

// What a token brings to one value head: its rows of 128 (in global or shared memory) and gates.  `conv`: the q, k and v rows in
// fp32 where the convolution ran in this kernel, else nullptr.
struct TokenRows {
  const __nv_bfloat16 *q, *k, *v, *z;
  const float (*conv)[kDk];
  float alpha, beta;
};
__device__ __forceinline__ float gate_alpha(float neg_a, float dtb, float a) {
  const float x = a + dtb;
  const float sp_x = x > 20.f ? x : log1pf(__expf(x));
  return __expf(neg_a * sp_x);
}
__device__ __forceinline__ float gate_beta(float b) { return 1.f / (1.f + __expf(-b)); }

// One token of one value head, by 256 threads that hold the head's state: thread (warp, lane) rows warp * 16 + 4 j + lane / 8 and
// float4 columns lane % 8 + 8 i.  `k_s`, `q_s`: 128 floats each of this warp; `red`: a float per warp, unlike that of the token
// before; `sync`: barrier of the 256 threads.
template <typename Sync>
__device__ __forceinline__ void token_step(const GdnParams& p, const TokenRows& in, float4 (&S)[kRowsPerThread][4], int t, int hv,
                                           int warp, int lane, float* k_s, float* q_s, float* red, Sync sync) {
  const int sub = lane >> 3, q8 = lane & 7;
  const float qscale = rsqrtf(static_cast<float>(kDk));
  // ---- per-warp copy of the normalised q, k of this token ----
  float kf[4], qf[4];
  if (in.conv != nullptr) {
    const float4 k4f = *reinterpret_cast<const float4*>(&in.conv[1][lane * 4]);
    const float4 q4f = *reinterpret_cast<const float4*>(&in.conv[0][lane * 4]);
    kf[0] = k4f.x; kf[1] = k4f.y; kf[2] = k4f.z; kf[3] = k4f.w;
    qf[0] = q4f.x; qf[1] = q4f.y; qf[2] = q4f.z; qf[3] = q4f.w;
  } else {
    const uint2 kr = *reinterpret_cast<const uint2*>(in.k + lane * 4);
    const uint2 qr = *reinterpret_cast<const uint2*>(in.q + lane * 4);
    const __nv_bfloat162* kp = reinterpret_cast<const __nv_bfloat162*>(&kr);
    const __nv_bfloat162* qp = reinterpret_cast<const __nv_bfloat162*>(&qr);
    kf[0] = __bfloat162float(kp[0].x); kf[1] = __bfloat162float(kp[0].y);
    kf[2] = __bfloat162float(kp[1].x); kf[3] = __bfloat162float(kp[1].y);
    qf[0] = __bfloat162float(qp[0].x); qf[1] = __bfloat162float(qp[0].y);
    qf[2] = __bfloat162float(qp[1].x); qf[3] = __bfloat162float(qp[1].y);
  }
  const float ssk = warp_sum(kf[0] * kf[0] + kf[1] * kf[1] + kf[2] * kf[2] + kf[3] * kf[3]);
  const float ssq = warp_sum(qf[0] * qf[0] + qf[1] * qf[1] + qf[2] * qf[2] + qf[3] * qf[3]);
  const float ik = rsqrtf(ssk + 1e-6f), iq = rsqrtf(ssq + 1e-6f) * qscale;
  __syncwarp();
  *reinterpret_cast<float4*>(k_s + lane * 4) = make_float4(kf[0] * ik, kf[1] * ik, kf[2] * ik, kf[3] * ik);
  *reinterpret_cast<float4*>(q_s + lane * 4) = make_float4(qf[0] * iq, qf[1] * iq, qf[2] * iq, qf[3] * iq);
  __syncwarp();
  float4 k4[4], q4[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    k4[i] = reinterpret_cast<const float4*>(k_s)[q8 + 8 * i];
    q4[i] = reinterpret_cast<const float4*>(q_s)[q8 + 8 * i];
  }

  const float alpha = in.alpha, beta = in.beta;

  // side-branch tokens (commit[t] == 0) read the state but do not change it:  o = alpha * (S q) + u * (k . q)
  const bool cm = p.commit == nullptr || p.commit[t] != 0;
  float kq = 0.f;
  if (!cm) {
#pragma unroll
    for (int i = 0; i < 4; ++i) kq += k4[i].x * q4[i].x + k4[i].y * q4[i].y + k4[i].z * q4[i].z + k4[i].w * q4[i].w;
    kq += __shfl_xor_sync(0xffffffffu, kq, 1);
    kq += __shfl_xor_sync(0xffffffffu, kq, 2);
    kq += __shfl_xor_sync(0xffffffffu, kq, 4);
  }
  float o[kRowsPerThread];
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < kRowsPerThread; ++j) {
    const int r = warp * 16 + j * 4 + sub;
    const float v = in.conv != nullptr ? in.conv[2][r] : __bfloat162float(in.v[r]);
    // same summation tree as the prefill kernels, so decode, prefill and replay stay bit-consistent
    float kp4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      kp4[i] = S[j][i].x * k4[i].x + S[j][i].y * k4[i].y + S[j][i].z * k4[i].z + S[j][i].w * k4[i].w;
    float ks = (kp4[0] + kp4[1]) + (kp4[2] + kp4[3]);
    ks += __shfl_xor_sync(0xffffffffu, ks, 1);
    ks += __shfl_xor_sync(0xffffffffu, ks, 2);
    ks += __shfl_xor_sync(0xffffffffu, ks, 4);
    const float u = beta * (v - alpha * ks);
    float oj = 0.f;
    if (cm) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        S[j][i].x = alpha * S[j][i].x + u * k4[i].x;
        S[j][i].y = alpha * S[j][i].y + u * k4[i].y;
        S[j][i].z = alpha * S[j][i].z + u * k4[i].z;
        S[j][i].w = alpha * S[j][i].w + u * k4[i].w;
        oj += S[j][i].x * q4[i].x + S[j][i].y * q4[i].y + S[j][i].z * q4[i].z + S[j][i].w * q4[i].w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        oj += S[j][i].x * q4[i].x + S[j][i].y * q4[i].y + S[j][i].z * q4[i].z + S[j][i].w * q4[i].w;
      oj *= alpha;
    }
    oj += __shfl_xor_sync(0xffffffffu, oj, 1);
    oj += __shfl_xor_sync(0xffffffffu, oj, 2);
    oj += __shfl_xor_sync(0xffffffffu, oj, 4);
    if (!cm) oj += u * kq;
    oj = __bfloat162float(__float2bfloat16(oj));  // bf16 boundary before the head norm
    o[j] = oj;
    if (q8 == 0) sq += oj * oj;
  }

  // ---- gated RMSNorm over the head's 128 outputs ----
  sq = warp_sum(sq);
  if (lane == 0) red[warp] = sq;
  sync();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) tot += red[w];
  const float inv = rsqrtf(tot / kDv + p.eps);
  float yq = 0.f;
  if (q8 < kRowsPerThread) {
    // lane q8 of each 8-lane group writes row j = q8 (all eight lanes hold all four o[j])
    float oj = o[0];
#pragma unroll
    for (int j = 1; j < kRowsPerThread; ++j) oj = (q8 == j) ? o[j] : oj;
    const int r = warp * 16 + q8 * 4 + sub;
    const float z = __bfloat162float(in.z[r]);
    const float nw = __bfloat162float(p.norm_w[r]);
    const float y = oj * inv * nw * (z / (1.f + __expf(-z)));
    p.out[static_cast<long long>(t) * (p.n_v_heads * kDv) + hv * kDv + r] = __float2bfloat16(y);
    yq = __bfloat162float(__float2bfloat16(y));
  }
  if (p.q_codes != nullptr) {
    // a warp owns sixteen consecutive outputs (rows warp * 16 ..): element e = 4 * q8 + sub sits in lane 8 * sub + q8
    float v[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = __shfl_sync(0xffffffffu, yq, (e & 3) * 8 + (e >> 2));
    if (lane == 0) nvfp4_store_block(v, t, hv * (kDv / 16) + warp, p.n_v_heads * kDv, p.q_codes, p.q_sf);
  }
}

__global__ void __launch_bounds__(kThreads, 2) gdn_recurrent_kernel(const GdnParams p) {
  __shared__ __align__(16) float k_s[kThreads / 32][kDk];
  __shared__ __align__(16) float q_s[kThreads / 32][kDk];
  __shared__ float red[2][kThreads / 32];
  __shared__ __align__(16) float conv_s[3][kDk];   // fused-conv decode: this CTA's q, k, v rows

  pdl_launch_next();
  // The step description (sequence ranges, state slots) is uploaded before the step's first kernel and the state
  // was last written by this kernel one step earlier, so neither depends on the kernel right before this one: the
  // 64 KB state load is issued BEFORE waiting for that kernel and overlaps its tail.  A replay pass reads
  // per-sequence ends that a kernel of this very step computed: it waits first.
  if (p.seq_end != nullptr) pdl_wait_prior();
  const int hv = blockIdx.x, seq = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane >> 3, q8 = lane & 7;
  const int hk = hv / (p.n_v_heads / p.n_qk_heads);
  const int t_begin = p.cu_seqlens[seq], t_end = p.seq_end != nullptr ? p.seq_end[seq] : p.cu_seqlens[seq + 1];
  const int ratio = p.n_v_heads / p.n_qk_heads;
  const bool fused = p.conv_w != nullptr;
  if (t_end <= t_begin) {
    pdl_wait_prior();   // every CTA waits before it leaves: a later kernel's wait then still implies all earlier ones
    if (fused && ratio > 1) cluster_sync_all();   // (the cluster's CTAs share the sequence: all of them are here)
    return;
  }
  const int slot = p.state_slot[seq];
  // fused conv: thread i < 128 owns q channel i and v channel i of this CTA's heads, thread 128 + i k channel i.  The
  // history is as old as the state (written one step ago): it is requested before the dependency wait as well.
  const int ci = threadIdx.x & 127;
  const int ch_a = threadIdx.x < 128 ? p.q_off + hk * kDk + ci : p.k_off + hk * kDk + ci;
  const int ch_v = p.v_off + hv * kDv + ci;
  float hist_a[3] = {0.f, 0.f, 0.f}, hist_v[3] = {0.f, 0.f, 0.f};
  __nv_bfloat16* st_a = nullptr;
  __nv_bfloat16* st_v = nullptr;
  if (fused) {
    st_a = p.conv_state + static_cast<long long>(slot) * 3 * p.conv_C + ch_a;
    st_v = p.conv_state + static_cast<long long>(slot) * 3 * p.conv_C + ch_v;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      hist_a[j] = __bfloat162float(st_a[j * p.conv_C]);
      if (threadIdx.x < 128) hist_v[j] = __bfloat162float(st_v[j * p.conv_C]);
    }
  }

  // thread's rows: r_j = warp*16 + j*4 + sub ; columns: float4 index q8 + 8*i
  float* sbase = p.state + (static_cast<long long>(slot) * p.n_v_heads + hv) * kDv * kDk;
  float4 S[kRowsPerThread][4];
#pragma unroll
  for (int j = 0; j < kRowsPerThread; ++j) {
    const int r = warp * 16 + j * 4 + sub;
#pragma unroll
    for (int i = 0; i < 4; ++i) S[j][i] = reinterpret_cast<const float4*>(sbase + r * kDk)[q8 + 8 * i];
  }
  const float neg_a = -__expf(p.A_log[hv]);
  const float dtb = p.dt_bias[hv];
  if (p.seq_end == nullptr) pdl_wait_prior();   // the projections of this step's tokens come from the previous kernel

  if (fused) {
    // four taps + SiLU on this CTA's 384 channels, rounded to bf16 like the separate kernel's output; then the roll
    const __nv_bfloat16* xrow = p.qkv + static_cast<long long>(t_begin) * p.ld_qkv;
    auto conv1 = [&](int ch, const float* hist, float x) {
      const uint2 wv = *reinterpret_cast<const uint2*>(p.conv_w + static_cast<long long>(ch) * 4);
      const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wv);
      float a = __bfloat162float(wp[0].x) * hist[0];
      a += __bfloat162float(wp[0].y) * hist[1];
      a += __bfloat162float(wp[1].x) * hist[2];
      a += __bfloat162float(wp[1].y) * x;
      a = a / (1.f + __expf(-a));
      return __bfloat162float(__float2bfloat16(a));
    };
    const float xa = __bfloat162float(xrow[ch_a]);
    conv_s[threadIdx.x < 128 ? 0 : 1][ci] = conv1(ch_a, hist_a, xa);
    float xv = 0.f;
    if (threadIdx.x < 128) {
      xv = __bfloat162float(xrow[ch_v]);
      conv_s[2][ci] = conv1(ch_v, hist_v, xv);
    }
    if (ratio > 1) cluster_sync_all();   // every value head of this key head has read the shared q / k history
    else __syncthreads();
    if (hv % ratio == 0) {
      st_a[0] = __float2bfloat16(hist_a[1]);
      st_a[p.conv_C] = __float2bfloat16(hist_a[2]);
      st_a[2 * p.conv_C] = __float2bfloat16(xa);
    }
    if (threadIdx.x < 128) {
      st_v[0] = __float2bfloat16(hist_v[1]);
      st_v[p.conv_C] = __float2bfloat16(hist_v[2]);
      st_v[2 * p.conv_C] = __float2bfloat16(xv);
    }
  }

  for (int t = t_begin; t < t_end; ++t) {
    const __nv_bfloat16* row = p.qkv + static_cast<long long>(t) * p.ld_qkv;
    const __nv_bfloat16* prow = p.proj + static_cast<long long>(t) * p.ld_proj;
    const TokenRows in = {row + p.q_off + hk * kDk, row + p.k_off + hk * kDk, row + p.v_off + hv * kDv, prow + p.z_off + hv * kDv,
                          fused ? conv_s : nullptr, gate_alpha(neg_a, dtb, __bfloat162float(prow[p.a_off + hv])),
                          gate_beta(__bfloat162float(prow[p.b_off + hv]))};
    token_step(p, in, S, t, hv, warp, lane, k_s[warp], q_s[warp], red[(t - t_begin) & 1], [] { __syncthreads(); });
  }

  if (p.write_state) {
#pragma unroll
    for (int j = 0; j < kRowsPerThread; ++j) {
      const int r = warp * 16 + j * 4 + sub;
#pragma unroll
      for (int i = 0; i < 4; ++i) reinterpret_cast<float4*>(sbase + r * kDk)[q8 + 8 * i] = S[j][i];
    }
  }
}

// Decode steps of many states: one CTA per SM walks its (sequence, value head) pairs with the states in a ring of three 64 KB
// buffers.  A state is contiguous, so it comes and goes by bulk copies that no thread waits in, and the token's rows come the
// same way: while one state is updated the last is written and the next are on their way.  (The kernel above has all its loads
// at a CTA's start and all its stores at its end.)  A state costs an SM 3.25 us, 40 bytes a ns of 44 that a copy moves.  Rows in
// shared memory are part of it: with the rows loaded by the threads, 1 us of latency after another, a state took 6.5 us.
constexpr int kRing = 3;
constexpr int kStateBytes = kDk * kDv * 4;
constexpr int kStreamThreads = kThreads + 32;
constexpr int kRowBytes = kDk * 2;                            // a token's q, k, v or z row of one head
constexpr int kSlotBytes = kStateBytes + 4 * kRowBytes;
constexpr int kStreamSmem = kRing * kSlotBytes + 128;

__device__ __forceinline__ void bulk_load(uint32_t smem, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(kStreamThreads, 1) gdn_stream_kernel(const GdnParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kRing], bar_done[kRing];
  __shared__ __align__(16) float k_s[kThreads / 32][kDk];
  __shared__ __align__(16) float q_s[kThreads / 32][kDk];
  __shared__ float red[2][kThreads / 32];
  __shared__ int abort_flag;
  pdl_launch_next();
  const uint32_t ring = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t* const ring_gen = smem_raw + (ring - smem_u32(smem_raw));
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int b = 0; b < kRing; ++b) {
      mbar_init(smem_u32(&bar_full[b]), 1);
      mbar_init(smem_u32(&bar_done[b]), kThreads / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_items = p.n_v_heads * p.n_seq;
  const int mine = (n_items - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  volatile int* abortp = &abort_flag;
  struct Item { int seq, hv, t0, t1; };
  auto item = [&](int n) {   // n-th of this CTA; a sequence without tokens keeps its state
    const int i = static_cast<int>(blockIdx.x) + n * static_cast<int>(gridDim.x);
    const int seq = i / p.n_v_heads;
    return Item{seq, i - seq * p.n_v_heads, p.cu_seqlens[seq], p.cu_seqlens[seq + 1]};
  };
  auto rows = [&](const Item& it, int t, const __nv_bfloat16** r) {   // q, k, v, z of token t
    const int hk = it.hv / (p.n_v_heads / p.n_qk_heads);
    const __nv_bfloat16* row = p.qkv + static_cast<long long>(t) * p.ld_qkv;
    r[0] = row + p.q_off + hk * kDk;
    r[1] = row + p.k_off + hk * kDk;
    r[2] = row + p.v_off + it.hv * kDv;
    r[3] = p.proj + static_cast<long long>(t) * p.ld_proj + p.z_off + it.hv * kDv;
  };
  if (warp == kThreads / 32) {
    // ---- copies, one thread.  As in the kernel above, states and the step's description depend on no kernel of this step ----
    if (lane == 0) {
      auto state = [&](const Item& it) {
        return p.state + (static_cast<long long>(p.state_slot[it.seq]) * p.n_v_heads + it.hv) * kDv * kDk;
      };
      int loaded = 0;
      auto load_state = [&](int n, const Item& it) {
        const uint32_t bar = smem_u32(&bar_full[n % kRing]);
        if (it.t1 > it.t0) {
          mbar_expect_tx(bar, kSlotBytes);
          bulk_load(ring + (n % kRing) * kSlotBytes, state(it), kStateBytes, bar);
        } else {
          mbar_arrive(bar);
        }
      };
      auto load_rows = [&](int n, const Item& it) {
        if (it.t1 > it.t0) {
          const __nv_bfloat16* r[4];
          rows(it, it.t0, r);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            bulk_load(ring + (n % kRing) * kSlotBytes + kStateBytes + i * kRowBytes, r[i], kRowBytes, smem_u32(&bar_full[n % kRing]));
        }
        loaded = n + 1;
      };
      const int primed = min(mine, kRing);
      for (int n = 0; n < primed; ++n) load_state(n, item(n));
      pdl_wait_prior();   // the projections of this step's tokens come from the previous kernel
      asm volatile("fence.proxy.async.global;" ::: "memory");
      for (int n = 0; n < primed; ++n) load_rows(n, item(n));
      for (int n = 0; n < mine; ++n) {
        if (!mbar_wait(smem_u32(&bar_done[n % kRing]), (n / kRing) & 1, abortp, p.status, kStatusStateDoneTimeout)) break;
        const Item it = item(n);
        if (it.t1 > it.t0) bulk_store(state(it), ring + (n % kRing) * kSlotBytes, kStateBytes);
        if (n + kRing < mine) {
          const Item next = item(n + kRing);
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the buffer has been read
          load_state(n + kRing, next);
          load_rows(n + kRing, next);
        }
      }
      if (*abortp) {   // unwinding: copies in flight land before the CTA leaves
        for (int j = max(0, loaded - kRing); j < loaded; ++j)
          for (uint32_t spin = 0; spin < (1u << 20); ++spin)
            if (mbar_try_wait(smem_u32(&bar_full[j % kRing]), (j / kRing) & 1)) break;
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    pdl_wait_prior();   // every warp waits before it leaves: a later kernel's wait then still implies all earlier ones
    return;
  }
  const int sub = lane >> 3, q8 = lane & 7;
  pdl_wait_prior();
  const auto sync = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
  // gates of an item's first token, fetched an item ahead
  float a, b, A_log, dtb;
  Item it = item(0);
  auto fetch_gates = [&](const Item& i) {
    const __nv_bfloat16* prow = p.proj + static_cast<long long>(min(i.t0, p.T - 1)) * p.ld_proj;
    a = __bfloat162float(prow[p.a_off + i.hv]);
    b = __bfloat162float(prow[p.b_off + i.hv]);
    A_log = p.A_log[i.hv];
    dtb = p.dt_bias[i.hv];
  };
  fetch_gates(it);
  int step = 0;
  for (int n = 0; n < mine; ++n) {
    uint8_t* const slot = ring_gen + (n % kRing) * kSlotBytes;
    __nv_bfloat16* const rows_s = reinterpret_cast<__nv_bfloat16*>(slot + kStateBytes);
    const float neg_a = -__expf(A_log), bias = dtb;
    float alpha = gate_alpha(neg_a, bias, a), beta = gate_beta(b);
    const Item cur = it;
    if (n + 1 < mine) {
      it = item(n + 1);
      fetch_gates(it);
    }
    // (one verdict for the warps: their barriers below are never divergent)
    const bool ok = mbar_wait(smem_u32(&bar_full[n % kRing]), (n / kRing) & 1, abortp, p.status, kStatusStateWaitTimeout);
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 256, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(all) : "r"(static_cast<uint32_t>(ok)) : "memory");
    if (!all) break;
    if (cur.t1 > cur.t0) {
      float4* const buf = reinterpret_cast<float4*>(slot) + (warp * 16 + sub) * (kDk / 4) + q8;
      float4 S[kRowsPerThread][4];
#pragma unroll
      for (int j = 0; j < kRowsPerThread; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[j][i] = buf[j * 4 * (kDk / 4) + 8 * i];
#pragma unroll 1
      for (int t = cur.t0; t < cur.t1; ++t, ++step) {
        if (t > cur.t0) {   // a longer sequence: its other tokens' rows by the threads themselves
          const __nv_bfloat16* r[4];
          rows(cur, t, r);
          sync();
          if (threadIdx.x < 4 * kDk / 8)
            reinterpret_cast<uint4*>(rows_s)[threadIdx.x] = reinterpret_cast<const uint4*>(r[threadIdx.x / (kDk / 8)])[threadIdx.x % (kDk / 8)];
          sync();
          const __nv_bfloat16* prow = p.proj + static_cast<long long>(t) * p.ld_proj;
          alpha = gate_alpha(neg_a, bias, __bfloat162float(prow[p.a_off + cur.hv]));
          beta = gate_beta(__bfloat162float(prow[p.b_off + cur.hv]));
        }
        const TokenRows in = {rows_s, rows_s + kDk, rows_s + 2 * kDk, rows_s + 3 * kDk, nullptr, alpha, beta};
        token_step(p, in, S, t, cur.hv, warp, lane, k_s[warp], q_s[warp], red[step & 1], sync);
      }
#pragma unroll
      for (int j = 0; j < kRowsPerThread; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) buf[j * 4 * (kDk / 4) + 8 * i] = S[j][i];
      fence_proxy_async_smem();
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&bar_done[n % kRing]));
  }
}

}  // namespace

const char* gdn_recurrent(const GdnParams& p, cudaStream_t stream, bool pdl) {
  if (p.T <= 0 || p.n_seq <= 0) return nullptr;
  if (p.n_v_heads % p.n_qk_heads) return "gdn_recurrent: value heads must be a multiple of qk heads";
  if ((p.q_off | p.k_off | p.ld_qkv) % 4) return "gdn_recurrent: q/k offsets must be multiples of 4";
  const int ratio = p.n_v_heads / p.n_qk_heads;
  if (p.conv_w != nullptr) {
    if (p.T != p.n_seq || p.seq_end != nullptr || p.commit != nullptr || !p.write_state)
      return "gdn_recurrent: the fused convolution is for plain decode steps (one token per sequence, state written)";
    if (p.conv_state == nullptr || p.conv_C <= 0 || ratio > 8) return "gdn_recurrent: bad fused-convolution arguments";
  } else if (p.T > p.n_seq && (p.v_off | p.z_off | p.ld_proj) % 4 == 0) {
    return gdn_prefill(p, stream, pdl);
  }
  cudaLaunchConfig_t cfg = {};
  // The streaming kernel from 6.5 states per SM: below, a CTA's first loads and last stores, which nothing overlaps, cost more
  // than the ring gives.  us, two CTAs per SM -> streamed, 48 value heads: 8 sequences 13.4 and 13.5, 16 23.0 and 23.7,
  // 24 33.0 -> 31.3, 32 44.5 -> 40.8 (4.9 TB/s), 64 81.4 -> 74.0, 128 154 -> 142 (5.7 TB/s; a copy moves 6.5); 32 heads: 24
  // sequences 23.2 and 23.7, 32 31.0 -> 28.5, 128 108 -> 97.  Bulk copies want 16-byte addresses.
  const bool streamed = p.conv_w == nullptr && p.seq_end == nullptr && p.commit == nullptr && p.write_state &&
                        2LL * p.n_v_heads * p.n_seq >= 13LL * device_sm_count() &&
                        (p.q_off | p.k_off | p.v_off | p.z_off) % 8 == 0 && p.ld_qkv % 8 == 0 && p.ld_proj % 8 == 0 &&
                        ((reinterpret_cast<uintptr_t>(p.state) | reinterpret_cast<uintptr_t>(p.qkv) |
                          reinterpret_cast<uintptr_t>(p.proj)) & 15) == 0;
  cfg.gridDim = dim3(p.n_v_heads, p.n_seq); cfg.blockDim = dim3(kThreads); cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.conv_w != nullptr && ratio > 1) {   // the value heads of one key head share its q / k history: one cluster
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = ratio;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  cudaError_t e;
  if (streamed) {
    static bool attr_set = false;
    if (!attr_set) {
      e = cudaFuncSetAttribute(gdn_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
      if (e != cudaSuccess) return cudaGetErrorString(e);
      attr_set = true;
    }
    const long long items = static_cast<long long>(p.n_v_heads) * p.n_seq;
    cfg.gridDim = dim3(static_cast<unsigned int>(items < device_sm_count() ? items : device_sm_count()));
    cfg.blockDim = dim3(kStreamThreads);
    cfg.dynamicSmemBytes = kStreamSmem;
    e = cudaLaunchKernelEx(&cfg, gdn_stream_kernel, p);
  } else {
    e = cudaLaunchKernelEx(&cfg, gdn_recurrent_kernel, p);
  }
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace nfb
