// mLSTM, token by token.  One thread-block cluster per (sequence, head); each CTA of the cluster owns VC value columns
// and keeps its slice of the matrix memory in registers over all tokens of the step: a thread holds four columns of
// every (256 / (VC / 4))-th row.  Per token: state update and both contractions (S^T q and n . q) in one pass over the
// registers, one shuffle + shared-memory reduction, then the head norm (sum of squares exchanged inside the cluster),
// the output gate and the store.  Steps with one token per sequence take a variant that streams the state.
#include "mlstm.h"

#include <cooperative_groups.h>

#include "../common/device.h"
#include "../common/elem.cuh"
#include "../common/launch.h"

namespace nfb {

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 256;

template <typename A, int VC, int R>
__global__ void __launch_bounds__(kThreads) mlstm_recurrent_kernel(const MlstmArgs p) {
  constexpr int kCg = VC / 4;                 // column groups
  constexpr int kRg = kThreads / kCg;         // row groups; a thread's rows are rg, rg + kRg, ...
  constexpr int kWarps = kThreads / 32;
  constexpr int kPartials = kCg <= 32 ? kWarps : kRg;   // partial sums per column group after the shuffles
  extern __shared__ __align__(16) float smem[];
  const int D = p.dim, V = p.vdim, H = p.n_heads;
  float* qs = smem;                           // [2][D]
  float* ks = qs + 2 * D;                     // [2][D]
  float* red = ks + 2 * D;                    // [kPartials][kCg][5]
  __shared__ float ss_part[2];                // sum of squares of this CTA's columns, by token parity
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = tid % kCg, rg = tid / kCg;
  const int n_cta = gridDim.x;                // cluster size along x
  const int v0 = blockIdx.x * VC;
  const int h = blockIdx.y, seq = blockIdx.z;
  const int col = v0 + c * 4;
  const bool col_ok = col < V;
  cg::cluster_group cluster = cg::this_cluster();

  pdl_launch_next();
  pdl_wait_prior();
  const int t_begin = p.cu_seqlens[seq], t_end = p.cu_seqlens[seq + 1];
  const long long slot = p.state_slot[seq];
  float* Sg = p.S + (slot * H + h) * D * V;
  float* ng = p.n + (slot * H + h) * D;
  float* mg = p.m + slot * H + h;
  float4 S[R];
  float n[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rg + i * kRg;
    S[i] = (r < D && col_ok) ? *reinterpret_cast<const float4*>(Sg + static_cast<long long>(r) * V + col)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
    n[i] = r < D ? ng[r] : 0.f;
  }
  float m = *mg;
  const float inv_cap = 1.f / p.gate_cap;
  const A* proj = static_cast<const A*>(p.proj);
  auto stage = [&](int t, int b) {
    const A* row = proj + t * p.ldp;
    for (int i = tid * 8; i < 2 * D; i += kThreads * 8) {
      float v[8];
      if (i < D) {
        load8(row + p.q_off + h * D + i, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] *= p.q_scale;
        store8(qs + b * D + i, v);
      } else {
        load8(row + p.k_off + h * D + i - D, v);
        store8(ks + b * D + i - D, v);
      }
    }
  };
  if (t_begin < t_end) stage(t_begin, 0);
  __syncthreads();
  for (int t = t_begin; t < t_end; ++t) {
    const int b = (t - t_begin) & 1;
    const float ig = p.gate_cap * tanhf(p.gates[t * p.ldg + p.i_off + h] * inv_cap);
    const float fr = p.gate_cap * tanhf(p.gates[t * p.ldg + p.f_off + h] * inv_cap);
    const float fg = fminf(fr, 0.f) - log1pf(expf(-fabsf(fr)));      // log sigmoid
    const float m_new = fmaxf(fg + m, ig);
    const float da = expf(fg + m - m_new), db = expf(ig - m_new);
    m = m_new;
    float v4[4] = {0.f, 0.f, 0.f, 0.f};
    if (col_ok) {
      const A* vr = proj + t * p.ldp + p.v_off + h * V + col;
#pragma unroll
      for (int j = 0; j < 4; ++j) v4[j] = elem_to_f(vr[j]);
    }
    if (t + 1 < t_end) stage(t + 1, b ^ 1);
    float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    const float* q = qs + b * D;
    const float* k = ks + b * D;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rg + i * kRg;
      if (r < D) {
        const float kb = k[r] * db, qr = q[r];
        S[i].x = fmaf(da, S[i].x, kb * v4[0]);
        S[i].y = fmaf(da, S[i].y, kb * v4[1]);
        S[i].z = fmaf(da, S[i].z, kb * v4[2]);
        S[i].w = fmaf(da, S[i].w, kb * v4[3]);
        n[i] = fmaf(da, n[i], kb);
        acc[0] = fmaf(S[i].x, qr, acc[0]);
        acc[1] = fmaf(S[i].y, qr, acc[1]);
        acc[2] = fmaf(S[i].z, qr, acc[2]);
        acc[3] = fmaf(S[i].w, qr, acc[3]);
        acc[4] = fmaf(n[i], qr, acc[4]);
      }
    }
    if constexpr (kCg < 32) {
#pragma unroll
      for (int e = 0; e < 5; ++e)
#pragma unroll
        for (int o = kCg; o < 32; o <<= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    }
    if (kCg >= 32 || lane < kCg) {
      float* dst = red + ((kCg <= 32 ? warp : rg) * kCg + c) * 5;
#pragma unroll
      for (int e = 0; e < 5; ++e) dst[e] = acc[e];
    }
    __syncthreads();
    // the first kCg threads (one warp at most) finish the token's columns
    float o4[4] = {0.f, 0.f, 0.f, 0.f};
    if (tid < 32) {
      float sq = 0.f;
      if (tid < kCg) {
        float den = 0.f;
        for (int w = 0; w < kPartials; ++w) {
          const float* src = red + (w * kCg + tid) * 5;
#pragma unroll
          for (int e = 0; e < 4; ++e) o4[e] += src[e];
          den += src[4];
        }
        const float inv = 1.f / (fmaxf(fabsf(den), expf(-m)) + 1e-6f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          o4[e] *= inv;
          sq += o4[e] * o4[e];
        }
      }
      sq = warp_sum(sq);
      if (tid == 0) ss_part[b] = sq;
    }
    float total = 0.f;
    if (n_cta > 1) {
      cluster.sync();
      if (tid < 32) {
        for (int r = 0; r < n_cta; ++r) total += *cluster.map_shared_rank(&ss_part[b], r);
      }
    } else {
      __syncthreads();
      total = ss_part[b];
    }
    if (tid < kCg && col_ok) {
      const float inv = 1.f / sqrtf(total / static_cast<float>(p.vdim_true) + p.eps);
      const A* gr = proj + t * p.ldp + p.g_off + h * V + col;
      A* dst = static_cast<A*>(p.out) + t * p.ldo + h * V + col;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        dst[e] = elem_from_f<A>(o4[e] * inv * p.norm[h * V + col + e] * sigmoid_of<A>(elem_to_f(gr[e])));
    }
  }
  // every CTA of the cluster has read n and m, and nobody still reads a neighbour's shared memory
  if (n_cta > 1) cluster.sync();
  if (!p.write_state) return;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rg + i * kRg;
    if (r < D && col_ok) *reinterpret_cast<float4*>(Sg + static_cast<long long>(r) * V + col) = S[i];
    if (r < D && c == 0 && blockIdx.x == 0) ng[r] = n[i];
  }
  if (tid == 0 && blockIdx.x == 0) *mg = m;
}

// One token per sequence: the state slice is streamed instead of kept (read, updated, written and contracted row by row),
// so few registers and many CTAs keep HBM busy.
template <typename A, int VC>
__global__ void __launch_bounds__(kThreads, 3) mlstm_decode_kernel(const MlstmArgs p) {
  constexpr int kCg = VC / 4, kRg = kThreads / kCg, kAhead = 8;
  constexpr int kPartials = kThreads / 32;
  extern __shared__ __align__(16) float smem[];
  const int D = p.dim, V = p.vdim, H = p.n_heads;
  float* qs = smem;            // [D]
  float* ks = qs + D;          // [D]
  float* ns = ks + D;          // [D] updated normaliser
  float* red = ns + D;         // [kPartials][kCg][5]
  __shared__ float ss_part;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = tid % kCg, rg = tid / kCg, n_cta = gridDim.x;
  const int h = blockIdx.y, seq = blockIdx.z, col = blockIdx.x * VC + c * 4;
  const bool col_ok = col < V;
  cg::cluster_group cluster = cg::this_cluster();
  pdl_launch_next();
  pdl_wait_prior();
  const int t = p.cu_seqlens[seq];
  const long long slot = p.state_slot[seq];
  float* Sg = p.S + (slot * H + h) * D * V + col;
  float* ng = p.n + (slot * H + h) * D;
  float* mg = p.m + slot * H + h;
  float4 S[kAhead];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int r = rg + (i0 + j) * kRg;
      if (r < D && col_ok) S[j] = __ldcs(reinterpret_cast<const float4*>(Sg + static_cast<long long>(r) * V));
    }
  };
  fetch(0);
  const float inv_cap = 1.f / p.gate_cap;
  const float ig = p.gate_cap * tanhf(p.gates[t * p.ldg + p.i_off + h] * inv_cap);
  const float fr = p.gate_cap * tanhf(p.gates[t * p.ldg + p.f_off + h] * inv_cap);
  const float fg = fminf(fr, 0.f) - log1pf(expf(-fabsf(fr)));      // log sigmoid
  const float m_old = *mg;
  const float m = fmaxf(fg + m_old, ig);
  const float da = expf(fg + m_old - m), db = expf(ig - m);
  const A* row = static_cast<const A*>(p.proj) + t * p.ldp;
  for (int i = tid; i < D; i += kThreads) {
    const float k = elem_to_f(row[p.k_off + h * D + i]) * db;
    qs[i] = elem_to_f(row[p.q_off + h * D + i]) * p.q_scale;
    ks[i] = k;
    ns[i] = fmaf(da, ng[i], k);
  }
  float v4[4] = {0.f, 0.f, 0.f, 0.f};
  if (col_ok) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v4[j] = elem_to_f(row[p.v_off + h * V + col + j]);
  }
  __syncthreads();
  float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  const int per = (D + kRg - 1) / kRg;
  for (int i0 = 0; i0 < per; i0 += kAhead) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int r = rg + (i0 + j) * kRg;
      if (r < D) {
        const float kb = ks[r], qr = qs[r];
        if (col_ok) {
          float4 s = S[j];
          s.x = fmaf(da, s.x, kb * v4[0]);
          s.y = fmaf(da, s.y, kb * v4[1]);
          s.z = fmaf(da, s.z, kb * v4[2]);
          s.w = fmaf(da, s.w, kb * v4[3]);
          if (p.write_state) __stcs(reinterpret_cast<float4*>(Sg + static_cast<long long>(r) * V), s);
          acc[0] = fmaf(s.x, qr, acc[0]);
          acc[1] = fmaf(s.y, qr, acc[1]);
          acc[2] = fmaf(s.z, qr, acc[2]);
          acc[3] = fmaf(s.w, qr, acc[3]);
        }
        acc[4] = fmaf(ns[r], qr, acc[4]);
      }
    }
    if (i0 + kAhead < per) fetch(i0 + kAhead);
  }
  if constexpr (kCg < 32) {
#pragma unroll
    for (int e = 0; e < 5; ++e)
#pragma unroll
      for (int o = kCg; o < 32; o <<= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
  }
  if (lane < kCg) {
    float* dst = red + (warp * kCg + c) * 5;
#pragma unroll
    for (int e = 0; e < 5; ++e) dst[e] = acc[e];
  }
  __syncthreads();
  float o4[4] = {0.f, 0.f, 0.f, 0.f};
  if (tid < 32) {
    float sq = 0.f;
    if (tid < kCg) {
      float den = 0.f;
      for (int w = 0; w < kPartials; ++w) {
        const float* src = red + (w * kCg + tid) * 5;
#pragma unroll
        for (int e = 0; e < 4; ++e) o4[e] += src[e];
        den += src[4];
      }
      const float inv = 1.f / (fmaxf(fabsf(den), expf(-m)) + 1e-6f);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o4[e] *= inv;
        sq += o4[e] * o4[e];
      }
    }
    sq = warp_sum(sq);
    if (tid == 0) ss_part = sq;
  }
  float total = 0.f;
  if (n_cta > 1) {
    cluster.sync();
    if (tid < 32)
      for (int r = 0; r < n_cta; ++r) total += *cluster.map_shared_rank(&ss_part, r);
  } else {
    __syncthreads();
    total = ss_part;
  }
  if (tid < kCg && col_ok) {
    const float inv = 1.f / sqrtf(total / static_cast<float>(p.vdim_true) + p.eps);
    const A* gr = row + p.g_off + h * V + col;
    A* dst = static_cast<A*>(p.out) + t * p.ldo + h * V + col;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      dst[e] = elem_from_f<A>(o4[e] * inv * p.norm[h * V + col + e] * sigmoid_of<A>(elem_to_f(gr[e])));
  }
  if (blockIdx.x == 0 && p.write_state) {   // (every CTA of the cluster has read n and m: it passed the cluster barrier)
    for (int i = tid; i < D; i += kThreads) ng[i] = ns[i];
    if (tid == 0) *mg = m;
  }
  if (n_cta > 1) cluster.sync();   // nobody leaves while a neighbour may still read its sum
}

// The same step where there are many states: one CTA per SM walks its (sequence, head) pairs, whole rows of the state in a ring of
// three buffers that bulk copies fill and empty while the rows in the third are updated.  A thread holds four columns and the
// sums of four of the sixteen row groups of the kernel above, whose order of summation (rows of a group, pairs of groups, slices
// of 64 columns) it keeps: the same bits, and a head's norm needs no cluster.
constexpr int kRing = 3, kChunkRows = 32, kStreamCols = 512, kStreamMaxDim = 512;
constexpr int kStreamWorkers = 512;
constexpr int kChunkBytes = kChunkRows * kStreamCols * 4;
constexpr int kSlices = kStreamCols / 64;
constexpr int kStreamSmem = kRing * kChunkBytes + 128;

__device__ __forceinline__ void bulk_load(uint32_t smem, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

template <typename A>
__global__ void __launch_bounds__(kStreamWorkers + 32, 1) mlstm_stream_kernel(const MlstmArgs p) {
  extern __shared__ __align__(16) uint8_t smem_b[];
  __shared__ __align__(8) uint64_t bar_full[kRing], bar_done[kRing];
  __shared__ float qs[kStreamMaxDim], ks[kStreamMaxDim], ns[kStreamMaxDim];
  __shared__ __align__(16) float part[8][kStreamCols];   // sums of two row groups each
  __shared__ float den_s[16], ss_s[kSlices];
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int D = p.dim, V = p.vdim, H = p.n_heads;
  const uint32_t ring = (smem_u32(smem_b) + 127u) & ~127u;
  uint8_t* const ring_gen = smem_b + (ring - smem_u32(smem_b));
  pdl_launch_next();
  if (tid == 0) {
    abort_flag = 0;
    for (int b = 0; b < kRing; ++b) {
      mbar_init(smem_u32(&bar_full[b]), 1);
      mbar_init(smem_u32(&bar_done[b]), kStreamWorkers / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* abortp = &abort_flag;
  const int chunks = (D + kChunkRows - 1) / kChunkRows;
  const int items = p.n_seq * H, mine = (items - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int total = mine * chunks;
  if (warp == kStreamWorkers / 32) {
    // ---- copies, one thread.  The call before may be a step of the same states, or a portion whose walk wrote them: it is waited
    //      for before anything is read ----
    if (lane == 0) {
      pdl_wait_prior();
      asm volatile("fence.proxy.async.global;" ::: "memory");   // bulk copies read what ordinary stores have written
      auto rows = [&](int n, uint32_t& bytes) {
        const int i = static_cast<int>(blockIdx.x) + n / chunks * static_cast<int>(gridDim.x), c = n % chunks;
        bytes = static_cast<uint32_t>(min(kChunkRows, D - c * kChunkRows)) * V * 4;
        return p.S + ((static_cast<long long>(p.state_slot[i / H]) * H + i % H) * D + c * kChunkRows) * V;
      };
      int loaded = 0;
      auto load = [&](int n) {
        uint32_t bytes;
        const float* src = rows(n, bytes);
        const uint32_t bar = smem_u32(&bar_full[n % kRing]);
        mbar_expect_tx(bar, bytes);
        bulk_load(ring + (n % kRing) * kChunkBytes, src, bytes, bar);
        loaded = n + 1;
      };
      for (int n = 0; n < min(total, kRing); ++n) load(n);
      for (int n = 0; n < total; ++n) {
        if (!mbar_wait(smem_u32(&bar_done[n % kRing]), (n / kRing) & 1, abortp, p.status, kStatusStateDoneTimeout)) break;
        uint32_t bytes;
        float* dst = rows(n, bytes);
        bulk_store(dst, ring + (n % kRing) * kChunkBytes, bytes);
        if (n + kRing < total) {
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the buffer has been read
          load(n + kRing);
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
  const auto sync = [] { asm volatile("bar.sync 1, 512;" ::: "memory"); };
  const int cg = tid & 127, quarter = tid >> 7, col = cg * 4;
  const bool col_ok = col < V;
  const float inv_cap = 1.f / p.gate_cap;
  pdl_wait_prior();
  int n = 0;
  for (int it = 0; it < mine; ++it) {
    const int i = static_cast<int>(blockIdx.x) + it * static_cast<int>(gridDim.x), seq = i / H, h = i % H;
    const int t = p.cu_seqlens[seq];
    const long long slot = p.state_slot[seq];
    float* ng = p.n + (slot * H + h) * D;
    float* mg = p.m + slot * H + h;
    const A* row = static_cast<const A*>(p.proj) + t * p.ldp;
    float v4[4] = {0.f, 0.f, 0.f, 0.f};
    if (col_ok) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v4[j] = elem_to_f(row[p.v_off + h * V + col + j]);
    }
    const float ig = p.gate_cap * tanhf(p.gates[t * p.ldg + p.i_off + h] * inv_cap);
    const float fr = p.gate_cap * tanhf(p.gates[t * p.ldg + p.f_off + h] * inv_cap);
    const float fg = fminf(fr, 0.f) - log1pf(expf(-fabsf(fr)));      // log sigmoid
    const float m_old = *mg;
    const float m = fmaxf(fg + m_old, ig);
    const float da = expf(fg + m_old - m), db = expf(ig - m);
    for (int r = tid; r < D; r += kStreamWorkers) {
      const float k = elem_to_f(row[p.k_off + h * D + r]) * db;
      qs[r] = elem_to_f(row[p.q_off + h * D + r]) * p.q_scale;
      ks[r] = k;
      ns[r] = fmaf(da, ng[r], k);
    }
    sync();
    if (tid < 16) {
      float d = 0.f;
      for (int r = tid; r < D; r += 16) d = fmaf(ns[r], qs[r], d);
      den_s[tid] = d;
    }
    float acc[4][4];
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[g][e] = 0.f;
    bool ok = true;
    for (int c = 0; c < chunks; ++c, ++n) {
      ok = mbar_wait(smem_u32(&bar_full[n % kRing]), (n / kRing) & 1, abortp, p.status, kStatusStateWaitTimeout);
      if (!ok) break;
      float* const buf = reinterpret_cast<float*>(ring_gen + (n % kRing) * kChunkBytes) + col;
      if (col_ok) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (c * kChunkRows + half * 16 >= D) break;
          float4 s[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) s[g] = *reinterpret_cast<const float4*>(buf + (half * 16 + quarter * 4 + g) * V);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int lr = half * 16 + quarter * 4 + g, r = c * kChunkRows + lr;
            const float kb = ks[r], qr = qs[r];
            s[g].x = fmaf(da, s[g].x, kb * v4[0]);
            s[g].y = fmaf(da, s[g].y, kb * v4[1]);
            s[g].z = fmaf(da, s[g].z, kb * v4[2]);
            s[g].w = fmaf(da, s[g].w, kb * v4[3]);
            *reinterpret_cast<float4*>(buf + lr * V) = s[g];
            acc[g][0] = fmaf(s[g].x, qr, acc[g][0]);
            acc[g][1] = fmaf(s[g].y, qr, acc[g][1]);
            acc[g][2] = fmaf(s[g].z, qr, acc[g][2]);
            acc[g][3] = fmaf(s[g].w, qr, acc[g][3]);
          }
        }
        fence_proxy_async_smem();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_done[n % kRing]));
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<float4*>(&part[2 * quarter + j][col]) =
          make_float4(acc[2 * j][0] + acc[2 * j + 1][0], acc[2 * j][1] + acc[2 * j + 1][1], acc[2 * j][2] + acc[2 * j + 1][2],
                      acc[2 * j][3] + acc[2 * j + 1][3]);
    // (a barrier, and one verdict for the warps: where rows did not come, neither n, m nor an output is written)
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 512, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(all) : "r"(static_cast<uint32_t>(ok)) : "memory");
    if (!all) break;
    for (int r = tid; r < D; r += kStreamWorkers) ng[r] = ns[r];
    if (tid == 0) *mg = m;
    float o4[4] = {0.f, 0.f, 0.f, 0.f};
    if (tid < 128) {
      float den = 0.f, sq = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
#pragma unroll
        for (int e = 0; e < 4; ++e) o4[e] += part[w][col + e];
        den += den_s[2 * w] + den_s[2 * w + 1];
      }
      const float inv = 1.f / (fmaxf(fabsf(den), expf(-m)) + 1e-6f);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o4[e] *= inv;
        sq += o4[e] * o4[e];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if ((lane & 15) == 0) ss_s[tid >> 4] = sq;
    }
    sync();
    if (tid < 128 && col_ok) {
      float sum = 0.f;
      for (int r = 0; r < (V + 63) / 64; ++r) sum += ss_s[r];
      const float inv = 1.f / sqrtf(sum / static_cast<float>(p.vdim_true) + p.eps);
      const A* gr = row + p.g_off + h * V + col;
      A* dst = static_cast<A*>(p.out) + t * p.ldo + h * V + col;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        dst[e] = elem_from_f<A>(o4[e] * inv * p.norm[h * V + col + e] * sigmoid_of<A>(elem_to_f(gr[e])));
    }
  }
}

template <typename A>
cudaError_t launch_stream(const MlstmArgs& a) {
  auto kern = mlstm_stream_kernel<A>;
  static bool attr_set = false;
  if (!attr_set) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const long long items = static_cast<long long>(a.n_seq) * a.n_heads;
  const unsigned int ctas = static_cast<unsigned int>(items < device_sm_count() ? items : device_sm_count());
  return launch_kernel(kern, dim3(ctas), dim3(kStreamWorkers + 32), kStreamSmem, a.stream, a.pdl, 1, a);
}

template <typename A, int VC>
cudaError_t launch_decode(const MlstmArgs& a) {
  const size_t smem = sizeof(float) * (3 * static_cast<size_t>(a.dim) + kThreads / 32 * (VC / 4) * 5);
  const int n_cta = (a.vdim + VC - 1) / VC;
  return launch_kernel(mlstm_decode_kernel<A, VC>, dim3(n_cta, a.n_heads, a.n_seq), dim3(kThreads), smem, a.stream, a.pdl, n_cta, a);
}

template <typename A, int VC, int R>
cudaError_t launch(const MlstmArgs& a) {
  constexpr int kCg = VC / 4;
  constexpr int kPartials = kCg <= 32 ? kThreads / 32 : kThreads / kCg;
  const size_t smem = sizeof(float) * (4 * static_cast<size_t>(a.dim) + kPartials * kCg * 5);
  const int n_cta = (a.vdim + VC - 1) / VC;
  return launch_kernel(mlstm_recurrent_kernel<A, VC, R>, dim3(n_cta, a.n_heads, a.n_seq), dim3(kThreads), smem, a.stream, a.pdl,
                       n_cta, a);
}

// Streams take the states of 256 KB and more (below, all stay with the clusters) where there are too many for the clusters' CTAs, 64
// columns each and three an SM, to be resident at once, or one for every second SM: below, a cluster reads a state faster than one
// CTA does.  A second round of states that is nearly empty costs a stream as much as a full one: from 320 columns on it still pays,
// heads of 192 and more then want the round two fifths full, and narrower ones, which leave most of a stream's threads without
// columns, no second round at all.  Behind a GEMM, us, clusters and streamed, by states:
//   256 x 512   48: 17.9, 18.0   52: 20.5, 18.2   148: 44.3, 28.4   160: 48.7, 42.2   296: 83.3, 52.6 (48 at the copy rate)
//   512 x 384   60: 25.5, 27.6   72: 35.9, 27.8   148: 59.8, 40.8   160: 63.8, 64.1   296: 107.9, 78.4
//   256 x 256   60: 13.6, 13.8   84: 14.4, 14.2   148: 24.0, 16.1   160: 25.0, 25.1   296: 40.2, 30.6
//   512 x 256   60: 23.0, 23.6   84: 25.0, 23.6   148: 43.5, 28.9   176: 46.6, 48.5   208: 50.7, 49.5
//   512 x 128   60: 19.1, 19.5   84: 20.2, 19.7   148: 22.6, 20.1   160: 23.1, 35.0   296: 38.1, 38.0   444: 48.3, 55.7
// Rounds of the 1 B layer-list decoder, twelve layers of four heads of 256 x 512: 12 sequences 1046 and 1105, 13 1146 -> 1111,
// 20 1346 -> 1245, 32 1525 -> 1347, 40 1734 -> 1712, 64 2137 -> 1931.
bool stream_pays(const MlstmArgs& a) {
  const long long states = static_cast<long long>(a.n_seq) * a.n_heads, sms = device_sm_count();
  if (static_cast<long long>(a.dim) * a.vdim * 4 < 256 * 1024) return false;
  const bool many = 10 * states * ((a.vdim + 63) / 64) >= 27 * sms || 2 * states >= sms;
  return many && (a.vdim >= 320 || states <= sms || (a.vdim >= 192 && 5 * states >= 7 * sms));
}

template <typename A>
const char* dispatch(const MlstmArgs& a) {
  cudaError_t e;
  if (a.one_token && a.write_state && a.vdim <= kStreamCols && a.dim <= kStreamMaxDim && stream_pays(a) &&
      (reinterpret_cast<uintptr_t>(a.S) & 15) == 0) {
    e = launch_stream<A>(a);
    return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
  }
  if (a.one_token) {
    e = a.vdim <= 8 * 64 ? launch_decode<A, 64>(a) : launch_decode<A, 128>(a);
    return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
  }
  if (a.vdim <= 8 * 64) {         // 16 row groups
    if (a.dim <= 64) e = launch<A, 64, 4>(a);
    else if (a.dim <= 128) e = launch<A, 64, 8>(a);
    else if (a.dim <= 256) e = launch<A, 64, 16>(a);
    else e = launch<A, 64, 32>(a);
  } else {                        // 8 row groups
    if (a.dim <= 128) e = launch<A, 128, 16>(a);
    else if (a.dim <= 256) e = launch<A, 128, 32>(a);
    else return "mlstm: value width above 512 needs a key width of at most 256";
  }
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace

const char* mlstm_recurrent(const MlstmArgs& a) {
  if (a.T <= 0 || a.n_seq <= 0) return nullptr;
  if (a.dim % 16 || a.vdim % 16 || a.dim > 512 || a.vdim > 1024)
    return "mlstm: head widths must be multiples of 16, at most 512 (keys) and 1024 (values)";
  if (a.ldp % 8 || a.ldo % 4 || a.q_off % 8 || a.k_off % 8 || a.v_off % 4 || a.g_off % 4) return "mlstm: misaligned rows";
  if (!(a.gate_cap > 0.f)) return "mlstm: the gate cap must be positive";
  if (a.n_seq > 65535 || a.n_heads > 65535) return "mlstm: too many sequences or heads";
  return a.f32 ? dispatch<float>(a) : dispatch<__nv_bfloat16>(a);
}

}  // namespace nfb
