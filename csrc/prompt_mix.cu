// What lies between the projections and the mixer of a gated full-attention layer, over prompts:
//   * attention_operands: per-head RMS norm (gain 1 + w) and partial rotation of queries and keys, and the rows of keys and values in the
//     store, where attention reads them;
//   * attention_gate:     the attention output times sigmoid of the gate that the query projection carries beside each head.
//
// Both are bound by memory traffic: every operand passes through once, 16 bytes a lane, one block per token (a warp takes several heads, whose
// loads are in flight together; with one head a warp and positions from 64-bit divisions the two took 174 and 96 us for 8192 tokens of 24
// heads of 256, and take 100 and 53).  As library calls
// they were 27 passes over the same rows (contiguous copies, conversions, norms, concatenations, store writes).
// A prompt of 333 tokens through Qwen3.5 0.8B took 1007 launches, 6.3 ms of them on the GPU, with library calls here and around the delta rule, and
// takes 276 launches and 2.8 ms with these, the fused passes of csrc/delta_rule.cu and csrc/delta_general.cu and products that share launches.
// Compiled without fast math; where a result is rounded to bf16 at once, the root and the gate's exponential and quotient are the hardware's approximations.
#include "common.cuh"

namespace tyr {

__device__ __forceinline__ void pm_load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = unpack_bf16x2(w[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
__device__ __forceinline__ void pm_store8(__nv_bfloat16* p, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

struct OperandArgs {
  const __nv_bfloat16 *q, *k, *v;        // rows of B * S tokens, head h at column h * head_stride
  long long q_row, k_row, v_row, q_head; // keys and values: heads D apart
  const __nv_bfloat16 *qw, *kw;          // gains [D]
  const float *cosT, *sinT;              // [S, half]: the tables' rows of these tokens
  __nv_bfloat16* q_out;                  // [B, S, H, D]
  __nv_bfloat16 *k_store, *v_store;      // [B, G, cap, D], written from slot `slot0` on
  int B, S, H, G, D, half, cap, slot0;
  float eps;
};

// Lane l keeps channels 8 l .. 8 l + 7 of a head (D <= 256), and the channels that rotate with them are half / 8 lanes away.
__global__ void __launch_bounds__(256, 3) attention_operands_kernel(OperandArgs a) {
  pdl_entry();
  const int lane = threadIdx.x & 31, d = lane * 8, shift = a.half >> 3;
  const int s = blockIdx.x, b = blockIdx.y;
  const long long row = static_cast<long long>(b) * a.S + s;
  const bool live = d < a.D, first = d < a.half, second = !first && d < 2 * a.half;
  const int partner = first ? lane + shift : second ? lane - shift : lane;
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  float c[8], sn[8];                       // cosine, and the sine with its partner's sign; channels that don't rotate: 1 and 0
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    c[j] = 1.f;
    sn[j] = 0.f;
  }
  if (first || second) {
    const long long at = static_cast<long long>(s) * a.half + (first ? d : d - a.half);      // half and d are multiples of 8
    const float4 c0 = *reinterpret_cast<const float4*>(a.cosT + at), c1 = *reinterpret_cast<const float4*>(a.cosT + at + 4);
    const float4 s0 = *reinterpret_cast<const float4*>(a.sinT + at), s1 = *reinterpret_cast<const float4*>(a.sinT + at + 4);
    const float sign = first ? -1.f : 1.f;
    c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    sn[0] = sign * s0.x; sn[1] = sign * s0.y; sn[2] = sign * s0.z; sn[3] = sign * s0.w;
    sn[4] = sign * s1.x; sn[5] = sign * s1.y; sn[6] = sign * s1.z; sn[7] = sign * s1.w;
  }
  const float inv_d = 1.f / a.D;
  auto turned = [&](uint4 in, const float (&gain)[8]) {
    const uint32_t words[4] = {in.x, in.y, in.z, in.w};
    float x[8], ss = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(words[j]);
      x[2 * j] = f.x;
      x[2 * j + 1] = f.y;
      ss += f.x * f.x + f.y * f.y;
    }
    const float rstd = rsqrtf(warp_sum(ss) * inv_d + a.eps);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      x[j] *= rstd * gain[j];
      const float other = __shfl_sync(0xffffffffu, x[j], partner);
      x[j] = x[j] * c[j] + other * sn[j];
    }
    return make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
  };
  float gain[8];
  auto load_gain = [&](const __nv_bfloat16* w) {
    pm_load8(w + (live ? d : 0), gain);
#pragma unroll
    for (int j = 0; j < 8; ++j) gain[j] += 1.f;
  };
  const int warp = threadIdx.x >> 5;
  constexpr int U = 3;                     // heads of a warp whose loads are in flight together
  const __nv_bfloat16* q_row = a.q + row * a.q_row + d;
  __nv_bfloat16* q_to = a.q_out + row * a.H * a.D + d;
  load_gain(a.qw);
  for (int h0 = warp; h0 < a.H; h0 += 8 * U) {
    uint4 in[U];
#pragma unroll
    for (int u = 0; u < U; ++u) in[u] = live && h0 + 8 * u < a.H ? *reinterpret_cast<const uint4*>(q_row + (h0 + 8 * u) * a.q_head) : none;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 out = turned(in[u], gain);
      if (live && h0 + 8 * u < a.H) *reinterpret_cast<uint4*>(q_to + (h0 + 8 * u) * a.D) = out;
    }
  }
  const long long slot = static_cast<long long>(b) * a.G * a.cap + a.slot0 + s;
  load_gain(a.kw);
  for (int h = warp; h < 2 * a.G; h += 8) {
    const bool is_v = h >= a.G;
    const int g = is_v ? h - a.G : h;
    const uint4 in = live ? *reinterpret_cast<const uint4*>((is_v ? a.v + row * a.v_row : a.k + row * a.k_row) + static_cast<long long>(g) * a.D + d) : none;
    const uint4 out = is_v ? in : turned(in, gain);
    if (live) *reinterpret_cast<uint4*>((is_v ? a.v_store : a.k_store) + (slot + static_cast<long long>(g) * a.cap) * a.D + d) = out;
  }
}

struct GateOutArgs {
  const __nv_bfloat16 *o, *gate;
  long long o_b, o_s, o_h, gate_row, gate_head;     // element strides of o [B, S, H, D] and gate [B * S, H, D]
  __nv_bfloat16* y;                                 // [B * S, H * D]
  long long rows;
  int S, H, D;
};

__global__ void __launch_bounds__(256) attention_gate_kernel(GateOutArgs a) {
  pdl_entry();
  const int vecs = a.D >> 3, n = a.H * vecs;
  const long long row = blockIdx.x;
  const __nv_bfloat16* o_row = a.o + row / a.S * a.o_b + row % a.S * a.o_s;
  const __nv_bfloat16* g_row = a.gate + row * a.gate_row;
  __nv_bfloat16* y_row = a.y + row * a.H * a.D;
#pragma unroll 3
  for (int i = threadIdx.x; i < n; i += 256) {
    const int h = i / vecs, d = i % vecs * 8;
    float o[8], g[8];
    pm_load8(o_row + h * a.o_h + d, o);
    pm_load8(g_row + h * a.gate_head + d, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = __fdividef(o[j], 1.f + __expf(-g[j]));     // a gate of -inf: 0, like the quotient
    pm_store8(y_row + i * 8, o);
  }
}

}  // namespace tyr

using namespace tyr;

// strides: q row, k row, v row, q head (elements); dims: B, S, H, G, D, half, cap, slot0.  The head size is a multiple of 8 up to 256, the rotated
// half a multiple of 8, all rows 16-byte aligned; slot0 + S <= cap.
extern "C" TYR_EXPORT int tyr_attention_operands(const void* q, const void* k, const void* v, const long long* strides, const void* qw, const void* kw,
                                                 const float* cosT, const float* sinT, void* q_out, void* k_store, void* v_store, const int* dims,
                                                 float eps, void* stream) {
  OperandArgs a{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, strides[0], strides[1], strides[2], strides[3],
                (const __nv_bfloat16*)qw, (const __nv_bfloat16*)kw, cosT, sinT, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_store, (__nv_bfloat16*)v_store,
                dims[0], dims[1], dims[2], dims[3], dims[4], dims[5], dims[6], dims[7], eps};
  if (a.B < 1 || a.B > 65535 || a.S < 1 || a.H < 1 || a.G < 1 || a.D < 8 || a.D > 256 || (a.D & 7) || a.half < 8 || (a.half & 7) || 2 * a.half > a.D) return -1;
  if (a.slot0 < 0 || a.slot0 + static_cast<long long>(a.S) > a.cap) return -2;
  if ((a.q_row | a.k_row | a.v_row | a.q_head) & 7) return -3;
  for (const void* p : {q, k, v, qw, kw, (const void*)cosT, (const void*)sinT, (const void*)q_out, (const void*)k_store, (const void*)v_store})
    if (p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15)) return -4;
  return (int)launch_dependent(attention_operands_kernel, dim3(a.S, a.B), dim3(256), 0, (cudaStream_t)stream, a);
}

// y [rows, H * D] = o * sigmoid(gate); o [rows / S, S, H, D] by (batch, token, head) strides, gate [rows, H, D] by (row, head) strides.
extern "C" TYR_EXPORT int tyr_attention_gate(const void* o, const void* gate, const long long* strides, void* y, long long rows, int S, int H, int D,
                                             void* stream) {
  if (rows < 1 || rows > 0x7fffffff || S < 1 || rows % S || H < 1 || D < 8 || (D & 7)) return -1;
  for (int i = 0; i < 5; ++i)
    if (strides[i] & 7) return -3;
  for (const void* p : {o, gate, (const void*)y})
    if (p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15)) return -4;
  const GateOutArgs a{(const __nv_bfloat16*)o, (const __nv_bfloat16*)gate, strides[0], strides[1], strides[2], strides[3], strides[4], (__nv_bfloat16*)y, rows, S, H, D};
  return (int)launch_dependent(attention_gate_kernel, dim3(static_cast<unsigned>(rows)), dim3(256), 0, (cudaStream_t)stream, a);
}
