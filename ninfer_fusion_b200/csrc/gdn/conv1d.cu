// Depthwise causal conv1d (4 taps) + SiLU for the GDN q/k/v channels, ragged
// batches, with the per-sequence 3-column history.  One thread owns a channel
// pair of one token and gathers its four taps from the projection rows (or the
// history for taps that fall before the sequence's first token of this call).
//
// Reference: include/ninfer/ops/causal_conv1d_silu.h, src/ops/kernel/causal_conv1d.cuh
// (state = last 3 columns, oldest -> newest).
#include "gdn.h"

#include "../common/ptx.cuh"
#include "../common/quotient.cuh"

namespace nfb {

namespace {

__device__ __forceinline__ float2 ld2(const __nv_bfloat16* p) {
  const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(p);
  return make_float2(__bfloat162float(v.x), __bfloat162float(v.y));
}

// input of sequence `seq` at token index tau (global index), channel pair c.
__device__ __forceinline__ float2 tap(const ConvParams& p, int tau, int seq_start, int slot, int c) {
  if (tau >= seq_start) return ld2(p.x + static_cast<long long>(tau) * p.ld_x + p.c_off + c);
  const int j = tau - seq_start + 3;  // 0..2
  return ld2(p.conv_state + (static_cast<long long>(slot) * 3 + j) * p.C + c);
}

// Token index `back` steps before t: along the draft tree's parent links while inside the window, then into the
// history (indices below seq_start).
__device__ __forceinline__ int ancestor(const ConvParams& p, int t, int back, int seq_start) {
  int cur = t;
  for (int i = 0; i < back; ++i) {
    if (p.parent != nullptr && cur >= seq_start) {
      const int par = p.parent[cur];
      cur = par >= 0 ? par : seq_start - 1;
    } else {
      cur -= 1;
    }
  }
  return cur;
}

__global__ void __launch_bounds__(128) conv1d_silu_kernel(const ConvParams p) {
  pdl_launch_next();
  pdl_wait_prior();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 2;
  const int t = blockIdx.x;
  if (c >= p.C) return;
  const int seq = p.token_seq[t];
  if (seq < 0) return;
  const int start = p.cu_seqlens[seq];
  const int slot = p.state_slot[seq];
  const uint4 wv = *reinterpret_cast<const uint4*>(p.w + static_cast<long long>(c) * 4);  // 2 channels x 4 taps
  const __nv_bfloat16* wp = reinterpret_cast<const __nv_bfloat16*>(&wv);
  float a0 = 0.f, a1 = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = tap(p, ancestor(p, t, 3 - j, start), start, slot, c);
    a0 += __bfloat162float(wp[j]) * x.x;
    a1 += __bfloat162float(wp[4 + j]) * x.y;
  }
  a0 = a0 / (1.f + __expf(-a0));
  a1 = a1 / (1.f + __expf(-a1));
  *reinterpret_cast<uint32_t*>(p.out + static_cast<long long>(t) * p.C + c) = pack_bf16x2(a0, a1);
}

// Prefill variant: one thread owns 4 channels of a run of 16 consecutive tokens and slides the three previous
// inputs through registers, so every input row is read once instead of four times, and the grid is T / 16 x C / 512 CTAs instead
// of T x C / 256.  Sequence boundaries inside a run reload the window from the new sequence's history.  Bound by what the SM can
// issue next to memory: two channels per multiplication, the quotient without a branch, four channels a thread so that seven CTAs
// fit (eight took 130 registers and three).  2048 tokens x 10240 channels, 13 us of traffic: 97 us with the per-token kernel, 36
// with one channel per instruction, 20 now; 1873 tokens of six sequences x 8192 36 -> 18.
constexpr int kConvRun = 16;

// two channels side by side: one instruction multiplies and adds both
struct Pair {
  unsigned long long v;
  __device__ __forceinline__ static Pair of(float x, float y) {
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(x), "f"(y));
    return p;
  }
  __device__ __forceinline__ void get(float& x, float& y) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
};
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  Pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ void unpack4(const uint2& u, Pair* v) {
  const uint32_t w[2] = {u.x, u.y};
#pragma unroll
  for (int i = 0; i < 2; ++i) v[i] = Pair::of(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}

// four channels from c on: taps, the last three inputs, one token
struct ConvLane {
  Pair w[4][2];     // [tap][channel pair]
  Pair win[3][2];
  __device__ __forceinline__ void load_taps(const ConvParams& p, int c) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {   // 4 channels x 4 taps = 32 bytes
      const uint4 u = *reinterpret_cast<const uint4*>(p.w + static_cast<long long>(c) * 4 + i * 8);
      const uint32_t a[2] = {u.x, u.y}, b[2] = {u.z, u.w};   // taps 0, 1 and 2, 3 of channels 2 i and 2 i + 1
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        w[2 * j][i] = Pair::of(__uint_as_float(a[j] << 16), __uint_as_float(b[j] << 16));
        w[2 * j + 1][i] = Pair::of(__uint_as_float(a[j] & 0xffff0000u), __uint_as_float(b[j] & 0xffff0000u));
      }
    }
  }
  __device__ __forceinline__ void open_window(const ConvParams& p, int c, int t, int s) {   // before token t of sequence s
    const int start = p.cu_seqlens[s];
    const int slot = p.state_slot[s];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int tau = t - 3 + j;
      unpack4(*reinterpret_cast<const uint2*>(tau >= start ? p.x + static_cast<long long>(tau) * p.ld_x + p.c_off + c
                                                           : p.conv_state + (static_cast<long long>(slot) * 3 + (tau - start + 3)) * p.C + c),
              win[j]);
    }
  }
  __device__ __forceinline__ void token(const ConvParams& p, int c, int t, const uint2& raw) {
    Pair cur[2];
    unpack4(raw, cur);
    uint32_t o[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float a, b;
      fma2(w[3][i], cur[i], fma2(w[2][i], win[2][i], fma2(w[1][i], win[1][i], mul2(w[0][i], win[0][i])))).get(a, b);
      o[i] = pack_bf16x2(gate_by(a, a), gate_by(b, b));
    }
    *reinterpret_cast<uint2*>(p.out + static_cast<long long>(t) * p.C + c) = make_uint2(o[0], o[1]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      win[0][i] = win[1][i];
      win[1][i] = win[2][i];
      win[2][i] = cur[i];
    }
  }
};
__device__ __forceinline__ uint2 conv_row(const ConvParams& p, int c, int t) {
  return *reinterpret_cast<const uint2*>(p.x + static_cast<long long>(t) * p.ld_x + p.c_off + c);
}

// A run with a boundary or an end in it: four rows at a time, and the window anew where a sequence starts.  (A function of its own:
// its registers do not weigh on the usual run.)
__device__ __noinline__ void conv_mixed_run(const ConvParams& p, int c, int t0, int t1) {
  ConvLane lane;
  lane.load_taps(p, c);
  int seq = -2;
#pragma unroll 1
  for (int t = t0; t < t1; t += 4) {
    uint2 raw[4];
    int of[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      of[i] = t + i < t1 ? p.token_seq[t + i] : -1;
      raw[i] = conv_row(p, c, min(t + i, t1 - 1));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (of[i] < 0) {
        seq = -2;
        continue;
      }
      if (of[i] != seq) {   // first token of this run, or a new sequence starts here
        seq = of[i];
        lane.open_window(p, c, t + i, seq);
      }
      lane.token(p, c, t + i, raw[i]);
    }
  }
}

__global__ void __launch_bounds__(128, 7) conv1d_silu_rows_kernel(const __grid_constant__ ConvParams p) {
  pdl_launch_next();
  pdl_wait_prior();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (c >= p.C) return;
  const int t0 = blockIdx.x * kConvRun, t1 = min(p.T, t0 + kConvRun);
  // A full run of one sequence, the usual case: nothing between the loads depends on the data, so eight rows are in flight at
  // a time (row by row behind the sequence test, a thread waited for sixteen loads in turn).
  const int first = p.token_seq[t0];
  bool one = first >= 0 && t1 - t0 == kConvRun;
  if (one) {
#pragma unroll
    for (int i = 1; i < kConvRun; ++i) one &= p.token_seq[t0 + i] == first;
  }
  if (!one) {
    conv_mixed_run(p, c, t0, t1);
    return;
  }
  uint2 raw[kConvRun / 2];
#pragma unroll
  for (int i = 0; i < kConvRun / 2; ++i) raw[i] = conv_row(p, c, t0 + i);
  ConvLane lane;
  lane.load_taps(p, c);
  lane.open_window(p, c, t0, first);
#pragma unroll
  for (int i = 0; i < kConvRun / 2; ++i) {
    const uint2 r = raw[i];
    raw[i] = conv_row(p, c, t0 + kConvRun / 2 + i);
    lane.token(p, c, t0 + i, r);
  }
#pragma unroll
  for (int i = 0; i < kConvRun / 2; ++i) lane.token(p, c, t0 + kConvRun / 2 + i, raw[i]);
}

__global__ void __launch_bounds__(128) conv1d_state_kernel(const ConvParams p) {
  pdl_launch_next();
  pdl_wait_prior();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 2;
  const int seq = blockIdx.x;
  if (c >= p.C) return;
  const int start = p.cu_seqlens[seq], end = p.seq_end != nullptr ? p.seq_end[seq] : p.cu_seqlens[seq + 1];
  if (end <= start) return;
  const int slot = p.state_slot[seq];
  // the new history = the last three inputs along the (accepted) path that ends at `last`
  const int last = p.last_token != nullptr ? p.last_token[seq] : end - 1;
  float2 v[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) v[j] = tap(p, ancestor(p, last, 2 - j, start), start, slot, c);
#pragma unroll
  for (int j = 0; j < 3; ++j)
    *reinterpret_cast<uint32_t*>(p.conv_state + (static_cast<long long>(slot) * 3 + j) * p.C + c) =
        pack_bf16x2(v[j].x, v[j].y);
}

// Decode fast path (exactly one token per sequence): conv, SiLU and the history roll in one
// launch.  The thread that owns (sequence, channel pair) is the only reader and writer of that
// history column, so there is no ordering problem.
__global__ void __launch_bounds__(128) conv1d_silu_decode_kernel(const ConvParams p) {
  pdl_launch_next();
  pdl_wait_prior();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 2;
  const int t = blockIdx.x;  // token index == sequence index
  if (c >= p.C) return;
  const int slot = p.state_slot[t];
  __nv_bfloat16* st = p.conv_state + static_cast<long long>(slot) * 3 * p.C + c;
  const uint4 wv = *reinterpret_cast<const uint4*>(p.w + static_cast<long long>(c) * 4);
  const __nv_bfloat16* wp = reinterpret_cast<const __nv_bfloat16*>(&wv);
  float2 x[4];
  x[0] = ld2(st);
  x[1] = ld2(st + p.C);
  x[2] = ld2(st + 2 * p.C);
  x[3] = ld2(p.x + static_cast<long long>(t) * p.ld_x + p.c_off + c);
  float a0 = 0.f, a1 = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a0 += __bfloat162float(wp[j]) * x[j].x;
    a1 += __bfloat162float(wp[4 + j]) * x[j].y;
  }
  a0 = a0 / (1.f + __expf(-a0));
  a1 = a1 / (1.f + __expf(-a1));
  *reinterpret_cast<uint32_t*>(p.out + static_cast<long long>(t) * p.C + c) = pack_bf16x2(a0, a1);
#pragma unroll
  for (int j = 0; j < 3; ++j)
    *reinterpret_cast<uint32_t*>(st + j * p.C) = pack_bf16x2(x[j + 1].x, x[j + 1].y);
}

}  // namespace

const char* causal_conv1d_silu(const ConvParams& p, cudaStream_t stream, bool pdl) {
  if (p.T <= 0) return nullptr;
  if (p.C % 2 || p.c_off % 2 || p.ld_x % 2) return "causal_conv1d_silu: channel counts/offsets must be even";
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(128); cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  cfg.gridDim = dim3(p.T, (p.C / 2 + 127) / 128);
  if (p.update_state && p.one_token_per_seq) {
    if (p.T != p.n_seq) return "causal_conv1d_silu: one_token_per_seq needs T == n_seq";
    cudaError_t e1 = cudaLaunchKernelEx(&cfg, conv1d_silu_decode_kernel, p);
    return e1 == cudaSuccess ? nullptr : cudaGetErrorString(e1);
  }
  cudaError_t e = cudaSuccess;
  const bool rows_ok = p.parent == nullptr && p.T >= 64 && p.C % 8 == 0 && p.c_off % 8 == 0 && p.ld_x % 8 == 0 &&
                       ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.out) |
                         reinterpret_cast<uintptr_t>(p.conv_state) | reinterpret_cast<uintptr_t>(p.w)) & 15) == 0;
  if (!p.state_only && rows_ok) {
    cfg.gridDim = dim3((p.T + kConvRun - 1) / kConvRun, (p.C / 4 + 127) / 128);
    e = cudaLaunchKernelEx(&cfg, conv1d_silu_rows_kernel, p);
    cfg.gridDim = dim3(p.T, (p.C / 2 + 127) / 128);
  } else if (!p.state_only) {
    e = cudaLaunchKernelEx(&cfg, conv1d_silu_kernel, p);
  }
  if (e != cudaSuccess) return cudaGetErrorString(e);
  if (p.update_state) {
    cfg.gridDim = dim3(p.n_seq, (p.C / 2 + 127) / 128);
    e = cudaLaunchKernelEx(&cfg, conv1d_state_kernel, p);
    if (e != cudaSuccess) return cudaGetErrorString(e);
  }
  return nullptr;
}

}  // namespace nfb
