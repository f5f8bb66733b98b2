// y[M, N] = x[M, K] @ W[N, K]^T (+ bias) for decode-sized M (1..32 rows): a weight-streaming kernel.  The product is bound
// by reading W once from HBM, so a CTA owns 16 weight rows and its 8 warps split K; every lane streams 16 bytes of two
// weight rows per step straight into mma.sync m16n8k16 A fragments (W rows are the M dimension of the tile, the tokens the
// N dimension; the reduction over K is order-free, so a lane's 8 consecutive channels serve as the fragment's k-slots and
// the activations are loaded with the same addressing).  Tokens beyond M load nothing.  Warp partials meet in shared memory.
//
// A matrix with too few 16-row tiles for the chip has its contraction split over the CTAs of a thread-block cluster, whose sums meet
// through distributed shared memory.  A decoding step is a chain of such products of 2 to 6 us each and is bound by the number of
// launches in it, so the split needs no second launch (and no workspace), and up to four matrices that read the same activations share a launch.
// Qwen3.5 0.8B, one row, 500 tokens of context: a step of 323 launches took 1275 us, one of 149 launches (the norms inside the products too, see
// sk_norm_rows) takes 943; the four products of a linear layer (6144, 2048, 16 and 16 rows of 1024) take 5.1 us in one launch.
//
// The reference sends these products to the library GEMM (cc/src/tyr.cpp:1003-1036).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "gates.cuh"

namespace tyr {

constexpr int kSkWarps = 8;

constexpr int kSkSegments = 4;
constexpr int kSkMaxSplits = 8;  // a portable cluster

// Matrices behind the first one that read the same activations: their 16-row tiles follow those of the first along gridDim.x.
struct SkinnySegments {
  int n;                                   // matrices in all, the first included
  int tile0[kSkSegments];                  // first tile of each
  const __nv_bfloat16* w[kSkSegments];
  __nv_bfloat16* y[kSkSegments];
  long long ldw[kSkSegments], ldy[kSkSegments];
  int N[kSkSegments];
};

struct SkinnyArgs {
  const __nv_bfloat16* x;      // [M, K], row stride ldx
  const __nv_bfloat16* w;      // [N, K], row stride ldw
  const __nv_bfloat16* w2;     // gated form only: the second matrix [N, K]; y = silu(x w^T) * (x w2^T)
  const __nv_bfloat16* bias;   // [N] or null
  __nv_bfloat16* y;            // [M, N], row stride ldy
  long long ldx, ldw, ldy;
  int M, N, K;
  long long hx, hw, hy;        // per-head form: elements from head to head
  int act;                     // 6: xIELU with factors act_a, act_b, 9: tanh-GELU times aux, as in csrc/gemm_tcgen05.cu; 0: none
  float act_a, act_b;
  const __nv_bfloat16* aux;    // [M, N], row stride ldaux
  long long ldaux;
  // NORM form: the activations are the RMS norm of x + resid (both [M, K], rows ldx and ldr apart; resid nullable) with gain norm_w (or 1 + norm_w);
  // the sum goes to resid_out [M, K] (nullable).
  const __nv_bfloat16 *resid, *norm_w;
  __nv_bfloat16* resid_out;
  long long ldr;
  float eps;
  int one_plus_w;
};

__device__ __forceinline__ float sk_act(float z, const SkinnyArgs& a, int tok, int row) {
  if (a.act == 9) return gelu_tanh(z) * __bfloat162float(a.aux[tok * a.ldaux + row]);
  return a.act == 6 ? fmaf(0.5f, z, z > 0.f ? a.act_a * z * z : a.act_b * (__expf(z) - 1.f - z)) : z;
}

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr long long kSkPrefetchBytes = 32LL << 20;   // L2 prefetch issued by one launch before its input is ready

// The norm in front of the products, taken again by every CTA: a launch of its own costs a decoding step about 2.5 us, reading the rows from the L2
// and one more reduction about 1.  A row belongs to 8 / (M rounded up to a power of two) warps; the sum is rounded to bf16 before the norm, like
// the norm kernel's.  -> xs [M][K + 8]
__device__ __forceinline__ void sk_norm_rows(const SkinnyArgs& a, __nv_bfloat16* xs, float* s_part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = a.M <= 1 ? 8 : a.M <= 2 ? 4 : a.M <= 4 ? 2 : 1;       // warps of a row
  const int row = warp / per, part = warp % per, nvec = a.K >> 3;
  const bool live = row < a.M;
  const bool first = blockIdx.x == 0 && blockIdx.y == 0 && a.resid_out != nullptr;
  auto unpack = [](uint4 u, float (&f)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 p = unpack_bf16x2(w[j]);
      f[2 * j] = p.x;
      f[2 * j + 1] = p.y;
    }
  };
  auto pack = [](const float (&f)[8]) {
    return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
  };
  float ss = 0.f;
  if (live)
#pragma unroll 4
    for (int v = part * 32 + lane; v < nvec; v += per * 32) {
      uint4 u = *reinterpret_cast<const uint4*>(a.x + row * a.ldx + v * 8);
      float f[8];
      unpack(u, f);
      if (a.resid != nullptr) {
        float r[8];
        unpack(*reinterpret_cast<const uint4*>(a.resid + row * a.ldr + v * 8), r);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += r[j];
        u = pack(f);
        unpack(u, f);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      *reinterpret_cast<uint4*>(xs + row * (a.K + 8) + v * 8) = u;
      if (first) *reinterpret_cast<uint4*>(a.resid_out + static_cast<long long>(row) * a.K + v * 8) = u;
    }
  ss = warp_sum(ss);
  if (lane == 0) s_part[warp] = ss;
  __syncthreads();
  if (live) {
    float t = 0.f;
    for (int i = 0; i < per; ++i) t += s_part[row * per + i];
    const float rstd = rsqrtf(t / a.K + a.eps);
#pragma unroll 4
    for (int v = part * 32 + lane; v < nvec; v += per * 32) {
      float f[8], w[8];
      unpack(*reinterpret_cast<const uint4*>(xs + row * (a.K + 8) + v * 8), f);
      unpack(__ldg(reinterpret_cast<const uint4*>(a.norm_w + v * 8)), w);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * (a.one_plus_w ? w[j] + 1.f : w[j]);
      *reinterpret_cast<uint4*>(xs + row * (a.K + 8) + v * 8) = pack(f);
    }
  }
  __syncthreads();
}

template <int TILES, bool GATED, bool NORM>        // token tiles of 8: M <= 8 * TILES; GATED: two matrices, SwiGLU epilogue
__global__ void __launch_bounds__(kSkWarps * 32) skinny_gemm_kernel(SkinnyArgs a, const __grid_constant__ SkinnySegments seg) {
  __shared__ float part[GATED ? 2 : 1][kSkWarps][TILES][16][8];
  extern __shared__ __align__(16) __nv_bfloat16 sk_rows[];         // NORM: [M][K + 8]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  int tile = blockIdx.x;
  if (!GATED && seg.n > 1) {
    int s = 0;
#pragma unroll
    for (int i = 1; i < kSkSegments; ++i) s = (i < seg.n && tile >= seg.tile0[i]) ? i : s;
    tile -= seg.tile0[s];
    a.w = seg.w[s];
    a.y = seg.y[s];
    a.ldw = seg.ldw[s];
    a.ldy = seg.ldy[s];
    a.N = seg.N[s];
  }
  const int row0 = tile * 16;
  // The weights are constants: while the kernel that produces `x` still runs (this one may already be resident, see
  // launch_dependent), pull the head of every weight row of this CTA into the L2.  The whole grid asks for at most
  // kSkPrefetchBytes, so what it brings in is still there when the loop below reads it.
  pdl_trigger();
  if (tid < (GATED ? 32 : 16) && (a.ldw & 7) == 0) {
    const int r = row0 + (tid & 15);
    const int chunks = a.K >> 5;
    const int c0 = static_cast<int>(static_cast<long long>(chunks) * blockIdx.y / gridDim.y);
    const int c1 = static_cast<int>(static_cast<long long>(chunks) * (blockIdx.y + 1) / gridDim.y);
    long long per_row = kSkPrefetchBytes / (static_cast<long long>(gridDim.x) * gridDim.y * (GATED ? 32 : 16));
    per_row = min(per_row & ~127LL, static_cast<long long>(c1 - c0) * 64);
    if (r < a.N && per_row >= 128)
      bulk_prefetch_l2((tid < 16 ? a.w : a.w2) + static_cast<long long>(r) * a.ldw + 32LL * c0, static_cast<uint32_t>(per_row));
  }
  pdl_wait();
  if constexpr (NORM) {
    __shared__ float s_part[kSkWarps];
    sk_norm_rows(a, sk_rows, s_part);
  }
  int r_lo = row0 + g, r_hi = row0 + g + 8;
  r_lo = r_lo < a.N ? r_lo : a.N - 1;            // clamped rows are not written
  r_hi = r_hi < a.N ? r_hi : a.N - 1;
  const __nv_bfloat16* w_lo = a.w + r_lo * a.ldw + 8 * t;
  const __nv_bfloat16* w_hi = a.w + r_hi * a.ldw + 8 * t;
  const __nv_bfloat16* v_lo = GATED ? a.w2 + r_lo * a.ldw + 8 * t : nullptr;
  const __nv_bfloat16* v_hi = GATED ? a.w2 + r_hi * a.ldw + 8 * t : nullptr;
  const __nv_bfloat16* xr[TILES];
  bool live[TILES];
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
    const int tok = 8 * i + g;
    live[i] = tok < a.M;
    xr[i] = NORM ? sk_rows + (live[i] ? tok : 0) * (a.K + 8) + 8 * t : a.x + (live[i] ? tok : 0) * a.ldx + 8 * t;
  }
  float acc[TILES][4], acc2[TILES][4];
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
    acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    acc2[i][0] = acc2[i][1] = acc2[i][2] = acc2[i][3] = 0.f;
  }

  const int chunks = a.K >> 5;                   // 32 channels per warp step
  const int c_lo = static_cast<int>(static_cast<long long>(chunks) * blockIdx.y / gridDim.y);
  const int c_hi = static_cast<int>(static_cast<long long>(chunks) * (blockIdx.y + 1) / gridDim.y);
#pragma unroll 4
  for (int c = c_lo + warp; c < c_hi; c += kSkWarps) {
    const uint4 lo = __ldcs(reinterpret_cast<const uint4*>(w_lo + 32 * c));    // streamed once: do not keep in cache
    const uint4 hi = __ldcs(reinterpret_cast<const uint4*>(w_hi + 32 * c));
    uint4 lo2 = make_uint4(0u, 0u, 0u, 0u), hi2 = lo2;
    if (GATED) {
      lo2 = __ldcs(reinterpret_cast<const uint4*>(v_lo + 32 * c));
      hi2 = __ldcs(reinterpret_cast<const uint4*>(v_hi + 32 * c));
    }
#pragma unroll
    for (int i = 0; i < TILES; ++i) {
      // The plain load keeps the gated form of 9 to 16 tokens at 69.4 us for 2 x 17408 x 5120, with __ldg beside the other form it takes 74.4; of 17 to 32
      // tokens 106 and 105.
      const uint4* xp = reinterpret_cast<const uint4*>(xr[i] + 32 * c);
      const uint4 xv = live[i] ? (NORM || (GATED && TILES == 2) ? *xp : __ldg(xp)) : make_uint4(0u, 0u, 0u, 0u);
      mma_16816(acc[i], lo.x, hi.x, lo.y, hi.y, xv.x, xv.y);
      mma_16816(acc[i], lo.z, hi.z, lo.w, hi.w, xv.z, xv.w);
      if (GATED) {
        mma_16816(acc2[i], lo2.x, hi2.x, lo2.y, hi2.y, xv.x, xv.y);
        mma_16816(acc2[i], lo2.z, hi2.z, lo2.w, hi2.w, xv.z, xv.w);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
    part[0][warp][i][g][2 * t] = acc[i][0];
    part[0][warp][i][g][2 * t + 1] = acc[i][1];
    part[0][warp][i][g + 8][2 * t] = acc[i][2];
    part[0][warp][i][g + 8][2 * t + 1] = acc[i][3];
    if (GATED) {
      part[1][warp][i][g][2 * t] = acc2[i][0];
      part[1][warp][i][g][2 * t + 1] = acc2[i][1];
      part[1][warp][i][g + 8][2 * t] = acc2[i][2];
      part[1][warp][i][g + 8][2 * t + 1] = acc2[i][3];
    }
  }
  __syncthreads();
  const int splits = gridDim.y;
  for (int idx = tid; idx < TILES * 8 * 16; idx += kSkWarps * 32) {
    const int tok = idx >> 4, r = idx & 15;        // consecutive threads write consecutive output columns
    const int row = row0 + r;
    float s = 0.f;
#pragma unroll
    for (int wp = 0; wp < kSkWarps; ++wp) s += part[0][wp][tok >> 3][r][tok & 7];
    if (!GATED && splits > 1) {
      part[0][0][tok >> 3][r][tok & 7] = s;        // read by this thread only so far: now the CTA's sum
      continue;
    }
    if (tok < a.M && row < a.N) {
      if (GATED) {
        float u = 0.f;
#pragma unroll
        for (int wp = 0; wp < kSkWarps; ++wp) u += part[1][wp][tok >> 3][r][tok & 7];
        a.y[tok * a.ldy + row] = __float2bfloat16(s / (1.f + __expf(-s)) * u);
      } else {
        if (a.bias) s += __bfloat162float(a.bias[row]);
        a.y[tok * a.ldy + row] = __float2bfloat16(sk_act(s, a, tok, row));
      }
    }
  }
  if (!GATED && splits > 1) {
    // the CTAs of the cluster hold one share of the contraction each: the first sums them in their order
    cluster_arrive();
    cluster_wait();
    if (blockIdx.y == 0) {
      for (int idx = tid; idx < TILES * 8 * 16; idx += kSkWarps * 32) {
        const int tok = idx >> 4, r = idx & 15, row = row0 + r;
        if (tok >= a.M || row >= a.N) continue;
        const uint32_t at = smem_u32(&part[0][0][tok >> 3][r][tok & 7]);
        float v[kSkMaxSplits], s = 0.f;
#pragma unroll
        for (int i = 0; i < kSkMaxSplits; ++i) {
          v[i] = 0.f;
          if (i < splits) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[i]) : "r"(mapa_shared(at, i)) : "memory");
        }
#pragma unroll
        for (int i = 0; i < kSkMaxSplits; ++i) s += v[i];
        if (a.bias) s += __bfloat162float(a.bias[row]);
        a.y[tok * a.ldy + row] = __float2bfloat16(sk_act(s, a, tok, row));
      }
    }
    cluster_arrive();                              // no CTA leaves while its sums are being read
    cluster_wait();
  }
}

// A small matrix of its own for each head: gridDim.y heads, a warp owns 16 rows of the head's matrix and its whole contraction.
template <int TILES>
__global__ void __launch_bounds__(kSkWarps * 32) skinny_heads_kernel(SkinnyArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int row0 = (blockIdx.x * kSkWarps + warp) * 16;
  pdl_trigger();
  if (row0 >= a.N) return;
  const __nv_bfloat16* w = a.w + blockIdx.y * a.hw;
  const __nv_bfloat16* w_lo = w + min(row0 + g, a.N - 1) * a.ldw + 8 * t;        // clamped rows are not written
  const __nv_bfloat16* w_hi = w + min(row0 + g + 8, a.N - 1) * a.ldw + 8 * t;
  constexpr int U = 4;                             // the weights need nothing from the kernel in front of this one
  const int chunks = a.K >> 5;
  uint4 lo[U], hi[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u < chunks) {
      lo[u] = __ldg(reinterpret_cast<const uint4*>(w_lo + 32 * u));
      hi[u] = __ldg(reinterpret_cast<const uint4*>(w_hi + 32 * u));
    }
  pdl_wait();
  const __nv_bfloat16* xr[TILES];
  bool live[TILES];
  float acc[TILES][4];
#pragma unroll
  for (int i = 0; i < TILES; ++i) {
    const int tok = 8 * i + g;
    live[i] = tok < a.M;
    xr[i] = a.x + blockIdx.y * a.hx + (live[i] ? tok : 0) * a.ldx + 8 * t;
    acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  }
  for (int c0 = 0; c0 < chunks; c0 += U) {
    uint4 xv[U][TILES];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < TILES; ++i) xv[u][i] = c0 + u < chunks && live[i] ? *reinterpret_cast<const uint4*>(xr[i] + 32 * (c0 + u)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c0 + u >= chunks) break;
#pragma unroll
      for (int i = 0; i < TILES; ++i) {
        mma_16816(acc[i], lo[u].x, hi[u].x, lo[u].y, hi[u].y, xv[u][i].x, xv[u][i].y);
        mma_16816(acc[i], lo[u].z, hi[u].z, lo[u].w, hi[u].w, xv[u][i].z, xv[u][i].w);
      }
      if (c0 + u + U < chunks) {
        lo[u] = __ldg(reinterpret_cast<const uint4*>(w_lo + 32 * (c0 + u + U)));
        hi[u] = __ldg(reinterpret_cast<const uint4*>(w_hi + 32 * (c0 + u + U)));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TILES; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int tok = 8 * i + 2 * t + (e & 1), row = row0 + g + (e >> 1) * 8;
      if (tok < a.M && row < a.N) a.y[blockIdx.y * a.hy + tok * a.ldy + row] = __float2bfloat16(acc[i][e]);
    }
}

}  // namespace tyr

// The kernels above read the activations through the L1: the eight CTAs of an SM walk the same rows of x.  A kernel with a
// large shared-memory footprint earlier in the stream leaves the SMs split in favour of shared memory, and a kernel that
// states no preference inherits that split.  Ask for just the shared memory that the resident CTAs need (registers and
// threads bound their number); the rest is L1.
template <int TILES, bool GATED>
static void skinny_set_carveout() {
  const int per_cta = (GATED ? 2 : 1) * tyr::kSkWarps * TILES * 16 * 8 * 4 + 1024;
  int ctas = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, tyr::skinny_gemm_kernel<TILES, GATED, false>, tyr::kSkWarps * 32, 0) != cudaSuccess ||
      ctas < 1)
    return;
  int pct = (ctas * per_cta * 100 + 227 * 1024 - 1) / (227 * 1024);
  if (pct > 100) pct = 100;
  cudaFuncSetAttribute(tyr::skinny_gemm_kernel<TILES, GATED, false>, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
}
static void skinny_prefer_l1() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (done[dev]) return;
  done[dev] = true;
  const char* v = getenv("TYR_SKINNY_CARVEOUT");
  if (v != nullptr && v[0] == '0') return;
  skinny_set_carveout<1, false>();
  skinny_set_carveout<2, false>();
  skinny_set_carveout<4, false>();
  skinny_set_carveout<1, true>();
  skinny_set_carveout<2, true>();
  skinny_set_carveout<4, true>();
}

// CTAs of a cluster that share the contraction of one 16-row tile: as many as stay resident at once beside the other tiles' (6 or 3 on an SM for up to 8 or 32
// tokens, 4 for 9 to 16 of which clusters find nine tenths), each with at least kSkSplitChannels channels, and none of a contraction that one CTA walks in few steps.  Weights
// from HBM, us at 1 / 2 / 3 / 4 / 8 CTAs: one row, 1024 x 3584 10.1 / 5.9 / 5.6 / 5.2 / 4.6, 3584 x 1024 3.7 / 4.5 / 4.7 / 6.9 / 11, 4096 x 12288 36.8 / 23.4 / 20.3 / 26.4 / 25.5,
// 5120 x 17408 52.1 / 34.1 / 44.6 / 36.4 / 42.2 (past one wave of CTAs it gets slower); 16 rows, 3072 x 2048 7.1 / 6.4 / 10.6 / 10.4 / 16.5; 32 rows, two matrices of
// 1024 x 5120 27.2 / 15.9 / 13.5 / 20.9 / 28.2.  Over 1 to 32 rows, 16 to 32000 columns and 512 to 17408 channels 0.8 % from the best on average, 25 % at most.
constexpr int kSkSplitChannels = 512, kSkSplitFrom = 1536;
static int skinny_splits(int row_ctas, int M, int K) {
  int splits = (M <= 8 ? 148 * 6 : M <= 16 ? 532 : 148 * 3) / row_ctas;
  if (M <= 16 && K < kSkSplitFrom) return 1;
  if (splits > K / kSkSplitChannels) splits = K / kSkSplitChannels;
  if (splits > tyr::kSkMaxSplits) splits = tyr::kSkMaxSplits;
  return splits < 1 ? 1 : splits;
}

template <int TILES, bool GATED, bool NORM = false>
static cudaError_t skinny_start(dim3 grid, cudaStream_t stream, const tyr::SkinnyArgs& a, const tyr::SkinnySegments& seg) {
  using namespace tyr;
  const size_t smem = NORM ? static_cast<size_t>(a.M) * (a.K + 8) * 2 : 0;
  if (grid.y == 1) return launch_dependent(skinny_gemm_kernel<TILES, GATED, NORM>, grid, dim3(kSkWarps * 32), smem, stream, a, seg);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kSkWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = grid.y; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = at; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, skinny_gemm_kernel<TILES, GATED, NORM>, a, seg);
}

static int skinny_launch(const tyr::SkinnyArgs& a, const tyr::SkinnySegments& seg, int row_ctas, int splits, void* stream) {
  using namespace tyr;
  if ((a.act != 0 && a.act != 6 && a.act != 9) || (a.act == 9) != (a.aux != nullptr)) return -4;
  if (a.M < 1 || a.M > 32 || a.K < 32 || (a.K & 31) || splits < 0 || splits > kSkMaxSplits) return -1;
  if (a.ldx & 7) return -2;                                          // 16-byte loads
  if (reinterpret_cast<uintptr_t>(a.x) & 15) return -3;
  for (int i = 0; i < seg.n; ++i) {
    if (seg.N[i] < 1) return -1;
    if (seg.ldw[i] & 7) return -2;
    if (reinterpret_cast<uintptr_t>(seg.w[i]) & 15) return -3;
  }
  const dim3 grid(row_ctas, splits > 0 ? splits : skinny_splits(row_ctas, a.M, a.K));
  const cudaStream_t st = (cudaStream_t)stream;
  skinny_prefer_l1();
  if (a.norm_w != nullptr) return (int)skinny_start<1, false, true>(grid, st, a, seg);
  return (int)(a.M <= 8 ? skinny_start<1, false>(grid, st, a, seg) : a.M <= 16 ? skinny_start<2, false>(grid, st, a, seg) : skinny_start<4, false>(grid, st, a, seg));
}

static int skinny_single(const void* x, const void* w, const void* bias, void* y, long long ldx, long long ldw, long long ldy, int M, int N, int K,
                         int act, float act_a, float act_b, void* stream, const void* aux = nullptr, long long ldaux = 0) {
  using namespace tyr;
  const SkinnyArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, nullptr, (const __nv_bfloat16*)bias, (__nv_bfloat16*)y, ldx, ldw, ldy, M, N, K,
                     0, 0, 0, act, act_a, act_b, (const __nv_bfloat16*)aux, ldaux};
  SkinnySegments seg{};
  seg.n = 1; seg.w[0] = a.w; seg.y[0] = a.y; seg.ldw[0] = ldw; seg.ldy[0] = ldy; seg.N[0] = N;
  return skinny_launch(a, seg, (N + 15) / 16, 0, stream);
}

static int skinny_many(tyr::SkinnyArgs a, int n, const void* const* w, void* const* y, const long long* ldw, const long long* ldy, const int* N, int splits,
                       void* stream) {
  using namespace tyr;
  if (n < 1 || n > kSkSegments) return -5;
  SkinnySegments seg{};
  seg.n = n;
  long long tiles = 0;
  for (int i = 0; i < n; ++i) {
    seg.tile0[i] = (int)tiles;
    seg.w[i] = (const __nv_bfloat16*)w[i];
    seg.y[i] = (__nv_bfloat16*)y[i];
    seg.ldw[i] = ldw[i];
    seg.ldy[i] = ldy[i];
    seg.N[i] = N[i];
    tiles += (N[i] + 15LL) / 16;
    if (tiles > 0x7fffffff) return -1;
  }
  a.w = seg.w[0];
  a.y = seg.y[0];
  a.ldw = ldw[0];
  a.ldy = ldy[0];
  a.N = N[0];
  return skinny_launch(a, seg, (int)tiles, splits, stream);
}

// Up to four matrices W[i] [N[i], K] that read the same x: y[i] = x W[i]^T in one launch.  `splits`: CTAs that share a contraction (0: by size).
extern "C" TYR_EXPORT int tyr_skinny_many_bf16(const void* x, long long ldx, int n, const void* const* w, void* const* y, const long long* ldw,
                                               const long long* ldy, const int* N, int M, int K, int splits, void* stream) {
  tyr::SkinnyArgs a{};
  a.x = (const __nv_bfloat16*)x; a.ldx = ldx; a.M = M; a.K = K;
  return skinny_many(a, n, w, y, ldw, ldy, N, splits, stream);
}

// The operand of the NORM forms: at most kSkNormNumbers of a batch's M <= 8 rows in a CTA's shared memory.
constexpr int kSkNormNumbers = 16384;
static int skinny_norm_args(tyr::SkinnyArgs& a, const void* x, const void* resid, const void* norm_w, void* resid_out, long long ldx, long long ldr, int M, int K,
                            float eps, int one_plus_w) {
  if (M < 1 || M > 8 || K < 32 || (K & 31) || M * (K + 8LL) > kSkNormNumbers || norm_w == nullptr) return -1;
  if ((ldx | ldr) & 7) return -2;
  for (const void* p : {x, resid, norm_w, (const void*)resid_out})
    if (reinterpret_cast<uintptr_t>(p) & 15) return -3;
  a.x = (const __nv_bfloat16*)x; a.resid = (const __nv_bfloat16*)resid; a.norm_w = (const __nv_bfloat16*)norm_w; a.resid_out = (__nv_bfloat16*)resid_out;
  a.ldx = ldx; a.ldr = ldr; a.M = M; a.K = K; a.eps = eps; a.one_plus_w = one_plus_w;
  return 0;
}

// The same of the RMS norm of x + resid (resid nullable; the sum goes to resid_out [M, K], nullable) with gain norm_w or 1 + norm_w.
extern "C" TYR_EXPORT int tyr_skinny_norm_many_bf16(const void* x, const void* resid, const void* norm_w, void* resid_out, long long ldx, long long ldr, int n,
                                                    const void* const* w, void* const* y, const long long* ldw, const long long* ldy, const int* N, int M,
                                                    int K, float eps, int one_plus_w, void* stream) {
  tyr::SkinnyArgs a{};
  const int rc = skinny_norm_args(a, x, resid, norm_w, resid_out, ldx, ldr, M, K, eps, one_plus_w);
  return rc ? rc : skinny_many(a, n, w, y, ldw, ldy, N, 0, stream);
}

// y [M, N] = silu(h wg^T) * (h wu^T) of the same norm h (both matrices with row stride ldw).
extern "C" TYR_EXPORT int tyr_skinny_norm_swiglu_bf16(const void* x, const void* resid, const void* norm_w, void* resid_out, long long ldx, long long ldr,
                                                      const void* wg, const void* wu, void* y, long long ldw, int M, int N, int K, float eps,
                                                      int one_plus_w, void* stream) {
  using namespace tyr;
  SkinnyArgs a{};
  const int rc = skinny_norm_args(a, x, resid, norm_w, resid_out, ldx, ldr, M, K, eps, one_plus_w);
  if (rc) return rc;
  if (N < 1) return -1;
  if (ldw & 7) return -2;
  if ((reinterpret_cast<uintptr_t>(wg) | reinterpret_cast<uintptr_t>(wu)) & 15) return -3;
  a.w = (const __nv_bfloat16*)wg; a.w2 = (const __nv_bfloat16*)wu; a.y = (__nv_bfloat16*)y;
  a.ldw = ldw; a.ldy = N; a.N = N;
  SkinnySegments seg{};
  seg.n = 1;
  return (int)skinny_start<1, true, true>(dim3((N + 15) / 16, 1), (cudaStream_t)stream, a, seg);
}

extern "C" TYR_EXPORT int tyr_skinny_gemm_bf16(const void* x, const void* w, const void* bias, void* y, long long ldx,
                                               long long ldw, long long ldy, int M, int N, int K, void* stream) {
  return skinny_single(x, w, bias, y, ldx, ldw, ldy, M, N, K, 0, 0.f, 0.f, stream);
}

// The same with an activation in the epilogue (6: xIELU, factors act_a above zero and act_b below).
extern "C" TYR_EXPORT int tyr_skinny_gemm_act_bf16(const void* x, const void* w, const void* bias, void* y, long long ldx, long long ldw,
                                                   long long ldy, int M, int N, int K, int act, float act_a, float act_b, void* stream) {
  return skinny_single(x, w, bias, y, ldx, ldw, ldy, M, N, K, act, act_a, act_b, stream);
}

// y[M, N] = gelu(x W^T) * aux (tanh form); aux [M, N] with row stride ldaux.
extern "C" TYR_EXPORT int tyr_skinny_gelu_mul_bf16(const void* x, const void* w, const void* aux, void* y, long long ldx, long long ldw,
                                                   long long ldaux, long long ldy, int M, int N, int K, void* stream) {
  return skinny_single(x, w, nullptr, y, ldx, ldw, ldy, M, N, K, 9, 0.f, 0.f, stream, aux, ldaux);
}

// A product of its own for each head: y[m, h, :N] = x[m, h, :K] @ W[h]^T for `heads` heads, rows (ldx, ldy) and heads (hx, hw, hy) apart
// by element strides.
extern "C" TYR_EXPORT int tyr_skinny_heads_bf16(const void* x, const void* w, void* y, long long ldx, long long hx, long long hw, long long ldw,
                                                long long ldy, long long hy, int heads, int M, int N, int K, void* stream) {
  using namespace tyr;
  if (M < 1 || M > 32 || N < 1 || K < 32 || (K & 31) || heads < 1 || heads > 65535) return -1;
  if ((ldx | ldw | hx | hw) & 7) return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return -3;
  SkinnyArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, nullptr, nullptr, (__nv_bfloat16*)y, ldx, ldw, ldy, M, N, K, hx, hw, hy, 0, 0.f, 0.f};
  const dim3 grid((N + 16 * kSkWarps - 1) / (16 * kSkWarps), heads), block(kSkWarps * 32);
  const cudaStream_t st = (cudaStream_t)stream;
  return (int)(M <= 8 ? launch_dependent(skinny_heads_kernel<1>, grid, block, 0, st, a)
                      : M <= 16 ? launch_dependent(skinny_heads_kernel<2>, grid, block, 0, st, a) : launch_dependent(skinny_heads_kernel<4>, grid, block, 0, st, a));
}

// y[M, N] = silu(x wg^T) * (x wu^T): the gate and up projections of a SwiGLU MLP for decode-sized M in one pass over both
// matrices (same row stride ldw), no intermediate tensors.
extern "C" TYR_EXPORT int tyr_skinny_swiglu_bf16(const void* x, const void* wg, const void* wu, void* y, long long ldx,
                                                 long long ldw, long long ldy, int M, int N, int K, void* stream) {
  using namespace tyr;
  if (M < 1 || M > 32 || N < 1 || K < 32 || (K & 31)) return -1;
  if ((ldx | ldw) & 7) return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(wg) | reinterpret_cast<uintptr_t>(wu)) & 15) return -3;
  SkinnyArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)wg, (const __nv_bfloat16*)wu, nullptr, (__nv_bfloat16*)y, ldx, ldw, ldy, M, N, K};
  SkinnySegments seg{};
  seg.n = 1;
  const dim3 grid((N + 15) / 16, 1);
  const cudaStream_t st = (cudaStream_t)stream;
  skinny_prefer_l1();
  return (int)(M <= 8 ? skinny_start<1, true>(grid, st, a, seg) : M <= 16 ? skinny_start<2, true>(grid, st, a, seg) : skinny_start<4, true>(grid, st, a, seg));
}
