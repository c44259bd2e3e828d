// Chunked (WY) gated delta rule for prefill: the recurrence over 64-token chunks as tensor-core matrix products.
//
// Per value head, with the chunk's incoming state S0 [dv, dk], cumulative log decays G_i (inclusive) and
// L2-normalised q, k:
//
//   A_ij = beta_i (k_i . k_j) exp(G_i - G_j)  (j < i),   X = (I + A)^-1
//   W = X (beta exp(G) k),  U = X (beta v),  P_ij = (q_i . k_j) exp(G_i - G_j) / sqrt(dk)  (j <= i)
//   u~ = U - W S0^T                                   (the per-token delta-rule updates, all at once)
//   O  = exp(G) (q S0^T) / sqrt(dk) + P u~
//   S1 = exp(G_C) S0 + (exp(G_C - G) u~)^T k
//
// which is algebraically the token-by-token rule `S = a S; u = beta (v - S k); S += u (x) k; o = S q / sqrt(dk)`.
//
// Three launches:
//   gdn_chunk_prepare  one CTA per (chunk, value head), all chunks in parallel: K K^T and Q K^T on mma.sync,
//                      the triangular inverse by forward substitution in two halves, W / U / P and the row scales into a
//                      workspace;
//   gdn_chunk_scan     one CTA per (sequence, value head, half or quarter of dv), sequential over the chunks: the state slice
//                      lives in MMA accumulator registers (fp32) of four warps, eight more load and write the output;
//                      the four products per chunk run on mma.sync out of a two-deep cp.async ring;
//   gdn_gated_norm     per (token, head) gated RMSNorm of the raw outputs in place.
//
// Operands of the products are bf16 (the inverse X as a hi + lo pair), accumulation and the state are fp32.
// mma.sync is used because the per-chunk products are 64 x 64 x 128 and run in a serial chain per head, where
// issue latency, not tensor throughput, sets the pace; a tcgen05 tile (M = 128) would be half empty.
//
// Reference: src/ops/linear_attention/gated_delta_net/chunked/{prepare_wy_wu,state_passing,output}.cuh
// (chunk 64, sub-block 16; same three-phase split).
#include "gdn.h"

#include <math_constants.h>

#include "../common/device.h"
#include "../common/ptx.cuh"
#include "../common/quotient.cuh"

namespace nfb {

namespace {

constexpr int kC = 64;          // tokens per chunk
constexpr int kD = 128;         // dk = dv
constexpr int kLdR = kD + 8;    // bf16 row pitch of [*, 128] tiles: 272 B, eight ldmatrix rows hit distinct banks
constexpr int kLdP = kC + 8;    // bf16 row pitch of [*, 64] tiles
constexpr int kLdA = kC + 4;    // fp32 row pitch of the A matrix (16-byte aligned rows)

struct WsView {
  __nv_bfloat16* W;   // [chunks * Hv, 64, 128]
  float* U;           // [chunks * Hv, 64, 128]
  __nv_bfloat16* P;   // [chunks * Hv, 64, 64]
  float* vec;         // [chunks * Hv, 3, 64]: q row scale, k row scale, exp(G_C) (broadcast)
};

struct ChunkParams {
  GdnParams g;
  WsView ws;
  int max_chunks;
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Chunk `ci` of the step (chunks are numbered sequence by sequence): its sequence, first token and token count.
__device__ __forceinline__ bool find_chunk(const int* cu, int n_seq, int ci, int& seq, int& t0, int& n) {
  int base = 0;
  for (int s = 0; s < n_seq; ++s) {
    const int b = cu[s], e = cu[s + 1];
    const int nc = (max(e - b, 0) + kC - 1) / kC;
    if (ci < base + nc) {
      seq = s;
      t0 = b + (ci - base) * kC;
      n = min(kC, e - t0);
      return true;
    }
    base += nc;
  }
  return false;
}

// ------------------------------------------------------------------------------------------------ prepare
struct PrepSmem {
  __nv_bfloat16 k[kC][kLdR];    // raw k rows (zero past the chunk's end); running sums; at last beta v
  __nv_bfloat16 q[kC][kLdR];    // raw q rows; once Q K^T is done, beta exp(G) k / |k|
  union {                       // A and the pieces of its inverse in fp32, then the inverse as a bf16 pair
    float a[kC][kLdA];
    struct {
      __nv_bfloat16 xh[kC][kLdP];
      __nv_bfloat16 xl[kC][kLdP];
    };
  };
  float g[kC], beta[kC], G[kC], rk[kC], rq[kC];
};

// Latency bound (short products and a serial inverse behind barriers; two warps per scheduler issued in 0.36 of the cycles),
// so what counts is how many chunks an SM works on at once and the length of the chain: the substitution's long rows summed by
// all warps, the row norms four rows at a time.  v is wanted last and comes into registers beside the end of the substitution, so
// that 54 KB of shared memory and 128 registers let four CTAs in.  Within a prompt's step of 2048 tokens: 48 heads 128 us with two
// CTAs and one thread per column, 105 with three; by itself 89 with three, 80 with four, 32 heads 66 and 57 (2.7 and 1.8 rounds
// of the grid).  Then shared memory was busy 60 % of the time; with norms that are reduced together, k scaled eight values at a
// time and even shares of the last products 73 and 51, one chunk 13 for 17.
__global__ void __launch_bounds__(128, 4) gdn_chunk_prepare_kernel(const ChunkParams cp) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  PrepSmem& sm = *reinterpret_cast<PrepSmem*>(smem_raw);
  const GdnParams& p = cp.g;
  int seq, t0, n_tok;
  if (!find_chunk(p.cu_seqlens, p.n_seq, blockIdx.x, seq, t0, n_tok)) return;
  const int hv = blockIdx.y;
  const int hk = hv / (p.n_v_heads / p.n_qk_heads);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long item = static_cast<long long>(blockIdx.x) * p.n_v_heads + hv;

  // ---- raw rows by cp.async (zero-filled past the chunk), gates by the first 64 threads ----
  for (int i = tid; i < 2 * kC * (kD / 8); i += blockDim.x) {
    const int which = i / (kC * (kD / 8)), r = (i / (kD / 8)) % kC, c = i % (kD / 8);
    const bool ok = r < n_tok;
    const __nv_bfloat16* src = p.qkv + static_cast<long long>(t0 + (ok ? r : 0)) * p.ld_qkv + (which ? p.q_off : p.k_off) + hk * kD + c * 8;
    __nv_bfloat16(*dst)[kLdR] = which ? sm.q : sm.k;
    cp_async_16(smem_u32(&dst[r][c * 8]), src, ok ? 16 : 0);
  }
  cp_async_commit();
  if (tid < kC) {
    float g = 0.f, beta = 0.f;
    if (tid < n_tok) {
      const __nv_bfloat16* prow = p.proj + static_cast<long long>(t0 + tid) * p.ld_proj;
      const float a = __bfloat162float(prow[p.a_off + hv]);
      const float b = __bfloat162float(prow[p.b_off + hv]);
      const float x = a + p.dt_bias[hv];
      const float sp = x > 20.f ? x : log1pf(__expf(x));
      g = -__expf(p.A_log[hv]) * sp;
      beta = 1.f / (1.f + __expf(-b));
    }
    sm.g[tid] = g;
    sm.beta[tid] = beta;
  }
  cp_async_wait<0>();
  __syncthreads();

  // ---- row norms (16 rows per warp, four at a time), inclusive scan of the log decays (warp 0) ----
#pragma unroll 1
  for (int r0 = warp * 16; r0 < warp * 16 + 16; r0 += 4) {
    float sk[4], sq[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint2 kw = *reinterpret_cast<const uint2*>(&sm.k[r0 + m][lane * 4]), qw = *reinterpret_cast<const uint2*>(&sm.q[r0 + m][lane * 4]);
      const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&kw);
      const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&qw);
      sk[m] = sq[m] = 0.f;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float2 kf = __bfloat1622float2(k2[e]), qf = __bfloat1622float2(q2[e]);
        sk[m] = fmaf(kf.y, kf.y, fmaf(kf.x, kf.x, sk[m]));
        sq[m] = fmaf(qf.y, qf.y, fmaf(qf.x, qf.x, sq[m]));
      }
    }
    // The sums of a warp's eight values, pairs of lanes 16, 8, 4, 2 and 1 apart as warp_sum adds them: after each of the first three
    // steps a lane goes on with the half of the values that its bit names.
    float s[8] = {sk[0], sk[1], sk[2], sk[3], sq[0], sq[1], sq[2], sq[3]};
#pragma unroll
    for (int n = 4, o = 16; n > 0; n /= 2, o /= 2) {
      const bool upper = lane & o;
#pragma unroll
      for (int m = 0; m < n; ++m) {
        const float other = __shfl_xor_sync(0xffffffffu, upper ? s[m] : s[m + n], o);
        s[m] = (upper ? s[m + n] : s[m]) + other;
      }
    }
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
    if ((lane & 3) == 0) (lane & 16 ? sm.rq : sm.rk)[r0 + (lane >> 2 & 3)] = rsqrtf(s[0] + 1e-6f);
  }
  if (warp == 0) {
    float a = sm.g[lane], b = sm.g[lane + 32];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) { a += ua; b += ub; }
    }
    const float total = __shfl_sync(0xffffffffu, a, 31);
    sm.G[lane] = a;
    sm.G[lane + 32] = b + total;
  }
  __syncthreads();

  // ---- K K^T and Q K^T for this warp's 16 rows; tiles above the diagonal are skipped ----
  const int row0 = lane >> 2, cq = lane & 3;
  {
    float kk[8][4], qk[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) { kk[n][j] = 0.f; qk[n][j] = 0.f; }
    const uint32_t ak_addr = smem_u32(&sm.k[warp * 16 + (lane & 7) + 8 * ((lane >> 3) & 1)][8 * (lane >> 4)]);
    const uint32_t aq_addr = smem_u32(&sm.q[warp * 16 + (lane & 7) + 8 * ((lane >> 3) & 1)][8 * (lane >> 4)]);
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      uint32_t a[4], b[4];
      ldsm_x4(ak_addr + ks * 32, a[0], a[1], a[2], a[3]);
      ldsm_x4(aq_addr + ks * 32, b[0], b[1], b[2], b[3]);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        if (np <= warp) {
          uint32_t c0, c1, c2, c3;
          ldsm_x4(smem_u32(&sm.k[np * 16 + (lane & 7) + 8 * (lane >> 4)][ks * 16 + 8 * ((lane >> 3) & 1)]), c0, c1, c2, c3);
          mma_bf16(kk[2 * np], a[0], a[1], a[2], a[3], c0, c1);
          mma_bf16(kk[2 * np + 1], a[0], a[1], a[2], a[3], c2, c3);
          mma_bf16(qk[2 * np], b[0], b[1], b[2], b[3], c0, c1);
          mma_bf16(qk[2 * np + 1], b[0], b[1], b[2], b[3], c2, c3);
        }
      }
    }
    const float qscale = rsqrtf(static_cast<float>(kD));
    __nv_bfloat16* Pg = cp.ws.P + item * (kC * kC);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (n / 2 > warp) {   // (of A nothing above the diagonal tile is read)
#pragma unroll
        for (int h = 0; h < 2; ++h) *reinterpret_cast<uint32_t*>(Pg + (warp * 16 + row0 + 8 * h) * kC + n * 8 + 2 * cq) = 0u;
        continue;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = warp * 16 + row0 + 8 * h;
        const int j = n * 8 + 2 * cq;
        float av[2], pv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int jj = j + e;
          const float dec = jj <= i ? __expf(sm.G[i] - sm.G[jj]) : 0.f;
          const float rkj = sm.rk[jj];
          av[e] = jj < i ? sm.beta[i] * sm.rk[i] * rkj * kk[n][2 * h + e] * dec : 0.f;
          pv[e] = jj <= i ? sm.rq[i] * rkj * qk[n][2 * h + e] * dec * qscale : 0.f;
        }
        *reinterpret_cast<float2*>(&sm.a[i][j]) = make_float2(av[0], av[1]);
        *reinterpret_cast<uint32_t*>(Pg + i * kC + j) = pack_bf16x2(pv[0], pv[1]);
      }
    }
  }
  __syncthreads();

  // ---- X = (I + A)^-1 by forward substitution, each entry's terms in the order of its row (four running sums, by column mod
  //      4).  Columns 0..31: warp 0 takes rows 0..31; then all warps take the terms of rows 32..63 with those; then warp 0 the
  //      rest of rows 32..63.  Columns 32..63 start at row 32 and are warp 1's meanwhile.  Lane c owns a column; the other two
  //      warps scale k, and beside the last part v comes into registers ----
  constexpr int kH = kC / 2;
  auto substitute = [&](int o, const float4* start, float* x) {   // rows o .. o + 31 and as many columns of A
#pragma unroll
    for (int i = 0; i < kH; ++i) {
      float acc[4] = {i == lane ? 1.f : 0.f, 0.f, 0.f, 0.f};
      if (start != nullptr) {
        const float4 s = start[i * kH + lane];
        acc[0] = s.x; acc[1] = s.y; acc[2] = s.z; acc[3] = s.w;
      }
#pragma unroll
      for (int j = 0; j < i; ++j) acc[j & 3] -= sm.a[o + i][o + j] * x[j];
      x[i] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
  };
  float x[kH];   // warps 0 and 1: rows of this lane's column in the diagonal half
  if (warp < 2) {
    substitute(warp * kH, nullptr, x);
    if (warp == 0) {   // (above the diagonal half: read below by all warps)
#pragma unroll
      for (int i = 0; i < kH; ++i) sm.a[i][kH + lane] = x[i];
    }
  } else {
#pragma unroll 4
    for (int i = tid - kC; i < kC * (kD / 8); i += 128 - kC) {
      const int r = i / (kD / 8), c = i % (kD / 8) * 8;
      const float sk = sm.beta[r] * __expf(sm.G[r]) * sm.rk[r];
      uint4 k = *reinterpret_cast<const uint4*>(&sm.k[r][c]);
      uint32_t* w = reinterpret_cast<uint32_t*>(&k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 kv = *reinterpret_cast<const __nv_bfloat162*>(&w[e]);
        w[e] = pack_bf16x2(__bfloat162float(kv.x) * sk, __bfloat162float(kv.y) * sk);
      }
      *reinterpret_cast<uint4*>(&sm.q[r][c]) = k;
    }
  }
  __syncthreads();
  float4* const sums = reinterpret_cast<float4*>(sm.k);   // [32 rows][32 columns] of four running sums, over the raw k rows
  static_assert(sizeof(float4) * kH * kH <= sizeof(sm.k), "the running sums lie over the k rows");
  {
    const int m0 = warp * 8;   // rows 32 + m0 .. + 7 and column `lane`
    float acc[8][4];
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][e] = 0.f;
#pragma unroll
    for (int j = 0; j < kH; j += 4) {
      float xc[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) xc[e] = sm.a[j + e][kH + lane];
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const float4 r = *reinterpret_cast<const float4*>(&sm.a[kH + m0 + m][j]);
        acc[m][0] -= r.x * xc[0];
        acc[m][1] -= r.y * xc[1];
        acc[m][2] -= r.z * xc[2];
        acc[m][3] -= r.w * xc[3];
      }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) sums[(m0 + m) * kH + lane] = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
  }
  __syncthreads();
  float x21[kH];
  constexpr int kVLoads = (kC * (kD / 8) + 95) / 96;   // 16-byte pieces of v per thread of warps 1..3
  uint4 v[kVLoads];
  if (warp == 0) {
    substitute(kH, sums, x21);
  } else {
#pragma unroll
    for (int j = 0; j < kVLoads; ++j) {
      const int i = j * 96 + tid - 32, r = i / (kD / 8), c = i % (kD / 8);
      v[j] = make_uint4(0, 0, 0, 0);
      if (r < n_tok)
        v[j] = *reinterpret_cast<const uint4*>(p.qkv + static_cast<long long>(t0 + r) * p.ld_qkv + p.v_off + hv * kD + c * 8);
    }
  }
  __syncthreads();   // (the bf16 pair lies over A, v over the running sums)
  if (warp != 0) {
#pragma unroll
    for (int j = 0; j < kVLoads; ++j) {
      const int i = j * 96 + tid - 32, r = i / (kD / 8), c = i % (kD / 8);
      if (r >= kC) break;
      const float sv = sm.beta[r];
      uint32_t* w = reinterpret_cast<uint32_t*>(&v[j]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 vv = *reinterpret_cast<const __nv_bfloat162*>(&w[e]);
        w[e] = pack_bf16x2(__bfloat162float(vv.x) * sv, __bfloat162float(vv.y) * sv);
      }
      *reinterpret_cast<uint4*>(&sm.k[r][c * 8]) = v[j];
    }
  }
  {
    auto put = [&](int i, int c, float v) {
      const __nv_bfloat16 hi = __float2bfloat16(v);
      sm.xh[i][c] = hi;
      sm.xl[i][c] = __float2bfloat16(v - __bfloat162float(hi));
    };
    // (the products below never read above the diagonal half)
    if (warp == 0) {
#pragma unroll
      for (int i = 0; i < kH; ++i) {
        put(i, lane, x[i]);
        put(kH + i, lane, x21[i]);
      }
    } else if (warp == 1) {
#pragma unroll
      for (int i = 0; i < kH; ++i) put(kH + i, kH + lane, x[i]);
    }
  }
  __syncthreads();

  // ---- W = X (beta exp(G) k^), U = X (beta v); X is lower triangular, so k-steps past the diagonal are skipped.  A warp has 32
  //      columns of all rows: with sixteen rows each the last warp had four times the first one's products ----
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    float acc[4][4][4];   // [row tile][8 columns]
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[m][n][j] = 0.f;
    __nv_bfloat16(*rhs)[kLdR] = pass == 0 ? sm.q : sm.k;
    const int xr = (lane & 7) + 8 * ((lane >> 3) & 1), xc = 8 * (lane >> 4);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t b[2][4];
#pragma unroll
      for (int np = 0; np < 2; ++np)
        ldsm_x4_trans(smem_u32(&rhs[kk * 16 + xr][warp * 32 + np * 16 + xc]), b[np][0], b[np][1], b[np][2], b[np][3]);
#pragma unroll
      for (int m = kk; m < 4; ++m) {
        uint32_t h[4], l[4];
        ldsm_x4(smem_u32(&sm.xh[m * 16 + xr][kk * 16 + xc]), h[0], h[1], h[2], h[3]);
        ldsm_x4(smem_u32(&sm.xl[m * 16 + xr][kk * 16 + xc]), l[0], l[1], l[2], l[3]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_bf16(acc[m][n], h[0], h[1], h[2], h[3], b[n / 2][n % 2 * 2], b[n / 2][n % 2 * 2 + 1]);
#pragma unroll
        for (int n = 0; n < 4; ++n) mma_bf16(acc[m][n], l[0], l[1], l[2], l[3], b[n / 2][n % 2 * 2], b[n / 2][n % 2 * 2 + 1]);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = m * 16 + row0 + 8 * h, j = warp * 32 + n * 8 + 2 * cq;
          if (pass == 0)
            *reinterpret_cast<uint32_t*>(cp.ws.W + item * (kC * kD) + i * kD + j) = pack_bf16x2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
          else
            *reinterpret_cast<float2*>(cp.ws.U + item * (kC * kD) + i * kD + j) = make_float2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
        }
  }

  // ---- row scales for the scan ----
  if (tid < kC) {
    float* vec = cp.ws.vec + item * (3 * kC);
    const float Gc = sm.G[kC - 1];
    vec[tid] = __expf(sm.G[tid]) * sm.rq[tid] * rsqrtf(static_cast<float>(kD));
    vec[kC + tid] = sm.rk[tid] * __expf(Gc - sm.G[tid]);
    vec[2 * kC + tid] = __expf(Gc);
  }
}

// ------------------------------------------------------------------------------------------------ scan
// The chunks of a sequence follow one another, so the time of one is the time of its longest chain: u~ = U - W S^T, then
// S = exp(G_C) S + u~^T K.  Warps 0-3 do nothing else (S in their registers); warps 4-7 compute the output rows Q S^T + P u~
// beside them, warps 8-11 load the next chunk's operands.  Two block barriers a chunk: operands and state are there, u~ is there.
// Within a prompt's step of 2048 tokens: 48 heads 112 us with eight warps that did both in turn, 106 with two groups of eight;
// by itself 91 with those, whose tiles of sixteen rows read 2560 wavefronts of shared memory per chunk (of 5400 cycles), and 84 with
// tiles of 32 rows (1660); 32 heads 63 and 58, in quarters of dv.  (Q S^T after u~, beside the state's update: 89.)
constexpr int kScanGroup = 128;                  // threads of the chain, of the output and of the loads
constexpr int kScanThreads = 3 * kScanGroup;

// DV: dv columns per CTA, 64 or 32
template <int DV>
struct ScanStage {
  __nv_bfloat16 w[kC][kLdR];
  __nv_bfloat16 q[kC][kLdR];
  __nv_bfloat16 k[kC][kLdR];
  __nv_bfloat16 p[kC][kLdP];
  float u[kC][DV + 4];
  float vec[3][kC];
};

template <int DV>
struct ScanSmem {
  ScanStage<DV> st[2];
  __nv_bfloat16 sb[DV][kLdR];    // state slice as bf16, [dv][dk]
  __nv_bfloat16 vn[kC][DV + 8];     // u~ (bf16)
  __nv_bfloat16 vnd[kC][DV + 8];      // exp(G_C - G) / |k| scaled u~
};

template <int DV>
__global__ void __launch_bounds__(kScanThreads, 1) gdn_chunk_scan_kernel(const ChunkParams cp) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  constexpr int kMt = DV / 16;   // row tiles of the state slice; also 8-column tiles per warp of a 64 x DV product
  ScanSmem<DV>& sm = *reinterpret_cast<ScanSmem<DV>*>(smem_raw);
  const GdnParams& p = cp.g;
  const int hv = blockIdx.x, slice = blockIdx.y, seq = blockIdx.z;
  const int hk = hv / (p.n_v_heads / p.n_qk_heads);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = lane >> 2, cq = lane & 3;
  const bool chain = warp < 4, loads = warp >= 8;
  const int mt = warp & 1, nh = (warp >> 1) & 1;   // products with 64 x DV outputs: half of the rows, half of the columns

  const int seq_b = p.cu_seqlens[seq], seq_e = p.cu_seqlens[seq + 1];
  if (seq_e <= seq_b) return;
  const int n_chunks = (seq_e - seq_b + kC - 1) / kC;
  int chunk0 = 0;
  for (int s = 0; s < seq; ++s) chunk0 += (max(p.cu_seqlens[s + 1] - p.cu_seqlens[s], 0) + kC - 1) / kC;

  const int ltid = tid - 2 * kScanGroup;     // of the loading warps
  auto load_stage = [&](int c, int stg) {
    ScanStage<DV>& st = sm.st[stg];
    const int t0 = seq_b + c * kC;
    const int n_tok = min(kC, seq_e - t0);
    const long long item = static_cast<long long>(chunk0 + c) * p.n_v_heads + hv;
    const __nv_bfloat16* Wg = cp.ws.W + item * (kC * kD);
    const __nv_bfloat16* Pg = cp.ws.P + item * (kC * kC);
    const float* Ug = cp.ws.U + item * (kC * kD) + slice * DV;
    const float* Vg = cp.ws.vec + item * (3 * kC);
    for (int i = ltid; i < kC * (kD / 8); i += kScanGroup) {
      const int r = i / (kD / 8), c8 = (i % (kD / 8)) * 8;
      cp_async_16(smem_u32(&st.w[r][c8]), Wg + r * kD + c8, 16);
      const bool ok = r < n_tok;
      const __nv_bfloat16* row = p.qkv + static_cast<long long>(t0 + (ok ? r : 0)) * p.ld_qkv + hk * kD + c8;
      cp_async_16(smem_u32(&st.q[r][c8]), row + p.q_off, ok ? 16 : 0);
      cp_async_16(smem_u32(&st.k[r][c8]), row + p.k_off, ok ? 16 : 0);
      if ((i % (kD / 8)) * 4 < DV) cp_async_16(smem_u32(&st.u[r][(i % (kD / 8)) * 4]), Ug + r * kD + (i % (kD / 8)) * 4, 16);
    }
    for (int i = ltid; i < kC * (kC / 8); i += kScanGroup) {
      const int r = i / (kC / 8), c8 = (i % (kC / 8)) * 8;
      cp_async_16(smem_u32(&st.p[r][c8]), Pg + r * kC + c8, 16);
    }
    if (ltid < 3 * kC / 4) cp_async_16(smem_u32(&st.vec[0][ltid * 4]), Vg + ltid * 4, 16);
  };

  if (loads) {
    load_stage(0, 0);
    cp_async_commit();
  }

  // state slice S[dv DV*slice ..][dk] in accumulator layout: warp w owns dk columns 32w..32w+31
  float* sbase = p.state + ((static_cast<long long>(p.state_slot[seq]) * p.n_v_heads + hv) * kD + slice * DV) * kD;
  float S[kMt][4][4];
  if (chain) {
#pragma unroll
    for (int mi = 0; mi < kMt; ++mi)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int dv = mi * 16 + row0 + 8 * h, dk = warp * 32 + n * 8 + 2 * cq;
          const float2 v = *reinterpret_cast<const float2*>(sbase + dv * kD + dk);
          S[mi][n][2 * h] = v.x;
          S[mi][n][2 * h + 1] = v.y;
          *reinterpret_cast<uint32_t*>(&sm.sb[dv][dk]) = pack_bf16x2(v.x, v.y);
        }
  }

  for (int c = 0; c < n_chunks; ++c) {
    const int stg = c & 1;
    ScanStage<DV>& st = sm.st[stg];
    if (loads) cp_async_wait<0>();
    __syncthreads();   // this chunk's operands and the bf16 state are visible; everyone is done with the other stage and vn / vnd
    if (loads) {
      if (c + 1 < n_chunks) {
        load_stage(c + 1, stg ^ 1);
        cp_async_commit();
      }
      __syncthreads();
      continue;
    }

    // ---- M1 = W S^T (chain) or O1 = Q S^T: rows 32 mt.., dv columns DV / 2 nh.. ----
    float acc[2][kMt][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < kMt; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[m][n][j] = 0.f;
    {
      const __nv_bfloat16(*left)[kLdR] = chain ? st.w : st.q;
      const uint32_t al = smem_u32(&left[mt * 32 + (lane & 7) + 8 * ((lane >> 3) & 1)][8 * (lane >> 4)]);
      const uint32_t bs = smem_u32(&sm.sb[nh * (DV / 2) + (lane & 7) + 8 * (lane >> 4)][8 * ((lane >> 3) & 1)]);
#pragma unroll
      for (int ks = 0; ks < kD / 16; ++ks) {
        uint32_t a[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m) ldsm_x4(al + m * 16 * kLdR * 2 + ks * 32, a[m][0], a[m][1], a[m][2], a[m][3]);
#pragma unroll
        for (int np = 0; np < kMt / 2; ++np) {
          uint32_t c0, c1, c2, c3;
          ldsm_x4(bs + np * 16 * kLdR * 2 + ks * 32, c0, c1, c2, c3);
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            mma_bf16(acc[m][2 * np], a[m][0], a[m][1], a[m][2], a[m][3], c0, c1);
            mma_bf16(acc[m][2 * np + 1], a[m][0], a[m][1], a[m][2], a[m][3], c2, c3);
          }
        }
      }
    }
    if (chain) {
      // ---- u~ = U - M1 (fp32), published as bf16 twice: plain and row-scaled for the state update ----
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < kMt; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = mt * 32 + m * 16 + row0 + 8 * h, col = nh * (DV / 2) + n * 8 + 2 * cq;
            const float2 u = *reinterpret_cast<const float2*>(&st.u[r][col]);
            const float v0 = u.x - acc[m][n][2 * h], v1 = u.y - acc[m][n][2 * h + 1];
            const float dk = st.vec[1][r];
            *reinterpret_cast<uint32_t*>(&sm.vn[r][col]) = pack_bf16x2(v0, v1);
            *reinterpret_cast<uint32_t*>(&sm.vnd[r][col]) = pack_bf16x2(v0 * dk, v1 * dk);
          }
    } else {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < kMt; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float dq = st.vec[0][mt * 32 + m * 16 + row0 + 8 * h];
            acc[m][n][2 * h] *= dq;
            acc[m][n][2 * h + 1] *= dq;
          }
    }
    __syncthreads();   // u~ is visible; everyone is done with the bf16 state

    if (chain) {
      // ---- S = exp(G_C) S + (scaled u~)^T K: all DV rows, dk columns 32 warp.. ----
      const float gamma = st.vec[2][0];
#pragma unroll
      for (int mi = 0; mi < kMt; ++mi)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) S[mi][n][j] *= gamma;
#pragma unroll
      for (int kk = 0; kk < kC / 16; ++kk) {
        uint32_t b[2][4];
#pragma unroll
        for (int np = 0; np < 2; ++np)
          ldsm_x4_trans(smem_u32(&st.k[kk * 16 + (lane & 7) + 8 * ((lane >> 3) & 1)][warp * 32 + np * 16 + 8 * (lane >> 4)]),
                        b[np][0], b[np][1], b[np][2], b[np][3]);
#pragma unroll
        for (int mi = 0; mi < kMt; ++mi) {
          uint32_t a[4];
          ldsm_x4_trans(smem_u32(&sm.vnd[kk * 16 + (lane & 7) + 8 * (lane >> 4)][mi * 16 + 8 * ((lane >> 3) & 1)]),
                        a[0], a[1], a[2], a[3]);
#pragma unroll
          for (int n = 0; n < 4; ++n) mma_bf16(S[mi][n], a[0], a[1], a[2], a[3], b[n / 2][n % 2 * 2], b[n / 2][n % 2 * 2 + 1]);
        }
      }
#pragma unroll
      for (int mi = 0; mi < kMt; ++mi)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int dv = mi * 16 + row0 + 8 * h, dk = warp * 32 + n * 8 + 2 * cq;
            *reinterpret_cast<uint32_t*>(&sm.sb[dv][dk]) = pack_bf16x2(S[mi][n][2 * h], S[mi][n][2 * h + 1]);
          }
    } else {
      // ---- O = O1 + P u~ ----
      const uint32_t ap = smem_u32(&st.p[mt * 32 + (lane & 7) + 8 * ((lane >> 3) & 1)][8 * (lane >> 4)]);
#pragma unroll
      for (int kk = 0; kk < kC / 16; ++kk) {
        uint32_t a[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m) ldsm_x4(ap + m * 16 * kLdP * 2 + kk * 32, a[m][0], a[m][1], a[m][2], a[m][3]);
        const int br = kk * 16 + (lane & 7) + 8 * ((lane >> 3) & 1);
#pragma unroll
        for (int np = 0; np < kMt / 2; ++np) {
          uint32_t c0, c1, c2, c3;
          ldsm_x4_trans(smem_u32(&sm.vn[br][nh * (DV / 2) + np * 16 + 8 * (lane >> 4)]), c0, c1, c2, c3);
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            mma_bf16(acc[m][2 * np], a[m][0], a[m][1], a[m][2], a[m][3], c0, c1);
            mma_bf16(acc[m][2 * np + 1], a[m][0], a[m][1], a[m][2], a[m][3], c2, c3);
          }
        }
      }
      const int t0 = seq_b + c * kC;
      const int n_tok = min(kC, seq_e - t0);
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = mt * 32 + m * 16 + row0 + 8 * h;
          if (r < n_tok) {
            __nv_bfloat16* dst = p.out + static_cast<long long>(t0 + r) * (p.n_v_heads * kD) + hv * kD + slice * DV + nh * (DV / 2) + 2 * cq;
#pragma unroll
            for (int n = 0; n < kMt; ++n)
              *reinterpret_cast<uint32_t*>(dst + n * 8) = pack_bf16x2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
          }
        }
    }
  }

  if (p.write_state && chain) {
#pragma unroll
    for (int mi = 0; mi < kMt; ++mi)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int dv = mi * 16 + row0 + 8 * h, dk = warp * 32 + n * 8 + 2 * cq;
          *reinterpret_cast<float2*>(sbase + dv * kD + dk) = make_float2(S[mi][n][2 * h], S[mi][n][2 * h + 1]);
        }
  }
}

// ------------------------------------------------------------------------------------------------ gated norm
// y = o * rsqrt(mean(o^2) + eps) * norm_w * silu(z), in place on `out`.  A warp takes four (token, head) rows and has all of
// their loads in flight: with one row, 512 bytes and a 64-bit division per warp, 2048 tokens of 48 heads (75 MB) took 24 us
// within a prompt's step, 21 so; of 32 heads 16 and 13.
constexpr int kNormRows = 4;

__global__ void __launch_bounds__(256) gdn_gated_norm_kernel(const GdnParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long n = static_cast<long long>(p.T) * p.n_v_heads;
  const long long idx0 = (static_cast<long long>(blockIdx.x) * 8 + warp) * kNormRows;
  if (idx0 >= n) return;
  __nv_bfloat16* o[kNormRows];
  uint2 ov[kNormRows], zv[kNormRows];
  int t = static_cast<int>(idx0 / p.n_v_heads), hv = static_cast<int>(idx0 - static_cast<long long>(t) * p.n_v_heads);
#pragma unroll
  for (int r = 0; r < kNormRows; ++r) {   // (a row past the end reads the last one and is not stored)
    o[r] = p.out + static_cast<long long>(t) * (p.n_v_heads * kD) + hv * kD + lane * 4;
    ov[r] = *reinterpret_cast<const uint2*>(o[r]);
    zv[r] = *reinterpret_cast<const uint2*>(p.proj + static_cast<long long>(t) * p.ld_proj + p.z_off + hv * kD + lane * 4);
    if (idx0 + r + 1 < n && ++hv == p.n_v_heads) {
      hv = 0;
      ++t;
    }
  }
  const uint2 wv = *reinterpret_cast<const uint2*>(p.norm_w + lane * 4);
  const auto unpack = [](const uint2& v, float* f) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      f[2 * i] = __bfloat162float(h[i].x);
      f[2 * i + 1] = __bfloat162float(h[i].y);
    }
  };
  float wf[4];
  unpack(wv, wf);
#pragma unroll
  for (int r = 0; r < kNormRows; ++r) {
    float of[4], zf[4], sq = 0.f;
    unpack(ov[r], of);
    unpack(zv[r], zf);
#pragma unroll
    for (int i = 0; i < 4; ++i) sq += of[i] * of[i];
    sq = warp_sum(sq);
    const float inv = rsqrtf(sq / kD + p.eps);
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = of[i] * inv * wf[i] * gate_by(zf[i], zf[i]);
    uint2 out;
    out.x = pack_bf16x2(y[0], y[1]);
    out.y = pack_bf16x2(y[2], y[3]);
    if (idx0 + r < n) *reinterpret_cast<uint2*>(o[r]) = out;
  }
}

}  // namespace

size_t gdn_chunked_workspace_bytes(int max_chunks, int n_v_heads) {
  const size_t items = static_cast<size_t>(max_chunks) * n_v_heads;
  return items * (kC * kD * 2 + kC * kD * 4 + kC * kC * 2 + 3 * kC * 4);
}

int gdn_chunked_max_chunks(int T, int n_seq) { return (T + kC - 1) / kC + n_seq; }

const char* gdn_chunked(const GdnParams& p, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  if (p.T <= 0 || p.n_seq <= 0) return nullptr;
  if (p.seq_end != nullptr || p.commit != nullptr) return "gdn_chunked: partial-sequence and tree passes use the recurrent kernels";
  if (p.n_v_heads % p.n_qk_heads) return "gdn_chunked: value heads must be a multiple of qk heads";
  if ((p.q_off | p.k_off | p.v_off | p.z_off) % 8 || p.ld_qkv % 8 || p.ld_proj % 4)
    return "gdn_chunked: row offsets and leading dimensions must be multiples of 8 elements";
  if ((reinterpret_cast<uintptr_t>(p.qkv) | reinterpret_cast<uintptr_t>(workspace)) & 15)
    return "gdn_chunked: inputs must be 16-byte aligned";
  if ((reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.norm_w)) & 7)
    return "gdn_chunked: proj / out / norm_w must be 8-byte aligned";
  ChunkParams cp;
  cp.g = p;
  cp.max_chunks = gdn_chunked_max_chunks(p.T, p.n_seq);
  if (workspace_bytes < gdn_chunked_workspace_bytes(cp.max_chunks, p.n_v_heads)) return "gdn_chunked: workspace too small";
  const size_t items = static_cast<size_t>(cp.max_chunks) * p.n_v_heads;
  uint8_t* base = static_cast<uint8_t*>(workspace);
  cp.ws.U = reinterpret_cast<float*>(base);
  base += items * kC * kD * 4;
  cp.ws.W = reinterpret_cast<__nv_bfloat16*>(base);
  base += items * kC * kD * 2;
  cp.ws.P = reinterpret_cast<__nv_bfloat16*>(base);
  base += items * kC * kC * 2;
  cp.ws.vec = reinterpret_cast<float*>(base);
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gdn_chunk_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(PrepSmem))) != cudaSuccess ||
        cudaFuncSetAttribute(gdn_chunk_scan_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(ScanSmem<64>))) != cudaSuccess ||
        cudaFuncSetAttribute(gdn_chunk_scan_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(ScanSmem<32>))) != cudaSuccess)
      return "gdn_chunked: cannot raise the shared-memory limit";
    attr_set = true;
  }
  gdn_chunk_prepare_kernel<<<dim3(cp.max_chunks, p.n_v_heads), 128, sizeof(PrepSmem), stream>>>(cp);
  // The scan is serial over the chunks and one CTA fills an SM: quarters of dv when all of them fit the GPU at once (32 heads:
  // 128 CTAs; 2048 tokens 102 us in halves, 71 in quarters, both before the chain had warps of its own), else halves (48 heads:
  // 96; quarters would run in two rounds).
  if (static_cast<long long>(p.n_v_heads) * 4 * p.n_seq <= device_sm_count())
    gdn_chunk_scan_kernel<32><<<dim3(p.n_v_heads, 4, p.n_seq), kScanThreads, sizeof(ScanSmem<32>), stream>>>(cp);
  else
    gdn_chunk_scan_kernel<64><<<dim3(p.n_v_heads, 2, p.n_seq), kScanThreads, sizeof(ScanSmem<64>), stream>>>(cp);
  const long long warps = static_cast<long long>(p.T) * p.n_v_heads;
  gdn_gated_norm_kernel<<<static_cast<unsigned int>((warps + 8 * kNormRows - 1) / (8 * kNormRows)), 256, 0, stream>>>(p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace nfb
