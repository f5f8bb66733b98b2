// Flux's tables of a denoising pass in one launch each: cosine and sine of every position (four axes of positions, text rows before
// image rows), and the sinusoidal embedding of the timesteps.  As library calls they were over a hundred launches of next to no work.
// Compiled without fast math: the angles reach 1000.
#include "common.cuh"

namespace tyr {

struct RopeTableArgs {
  const long long* ids[2];     // [B, rows, 4] of text and image
  int rows[2];
  int axis_end[4];             // pairs up to and including each axis
  int B, half;
  float log_theta;
  float *cosv, *sinv;          // [B, rows[0] + rows[1], half]
};

__global__ void __launch_bounds__(256) flux_rope_table_kernel(RopeTableArgs a) {
  pdl_entry();
  const int S = a.rows[0] + a.rows[1];
  const long long total = static_cast<long long>(a.B) * S * a.half;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const int j = static_cast<int>(i % a.half);
    const long long bs = i / a.half;
    const int s = static_cast<int>(bs % S);
    const long long b = bs / S;
    int ax = 0;
    while (j >= a.axis_end[ax]) ++ax;
    const int first = ax ? a.axis_end[ax - 1] : 0, n = a.axis_end[ax] - first;
    const long long id = s < a.rows[0] ? a.ids[0][(b * a.rows[0] + s) * 4 + ax] : a.ids[1][(b * a.rows[1] + s - a.rows[0]) * 4 + ax];
    const float angle = static_cast<float>(id) * expf(static_cast<float>(j - first) * (1.f / n) * -a.log_theta);
    float sn, cs;
    sincosf(angle, &sn, &cs);
    a.cosv[i] = cs;
    a.sinv[i] = sn;
  }
}

__global__ void __launch_bounds__(256) timestep_embedding_kernel(const float* __restrict__ t, __nv_bfloat16* __restrict__ out, int B, int dim, float factor,
                                                                 float log_period) {
  pdl_entry();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= B * dim) return;
  const int half = dim / 2, c = i % dim, j = c < half ? c : c - half;
  const float angle = t[i / dim] * factor * expf(-log_period * static_cast<float>(j) / half);
  out[i] = __float2bfloat16(c < half ? cosf(angle) : c < 2 * half ? sinf(angle) : 0.f);
}

}  // namespace tyr

using namespace tyr;

// rows: of text and image; axis_dims: pairs of each axis (all positive, `half` in all).
extern "C" TYR_EXPORT int tyr_flux_rope_table(const void* txt_ids, const void* img_ids, const int* rows, const int* axis_dims, int B, int half,
                                              float log_theta, float* cosv, float* sinv, void* stream) {
  RopeTableArgs a{{(const long long*)txt_ids, (const long long*)img_ids}, {rows[0], rows[1]}, {0, 0, 0, 0}, B, half, log_theta, cosv, sinv};
  int end = 0;
  for (int i = 0; i < 4; ++i) {
    if (axis_dims[i] <= 0) return -1;
    a.axis_end[i] = end += axis_dims[i];
  }
  if (end != half || B < 1 || rows[0] < 0 || rows[1] < 0 || rows[0] + rows[1] < 1) return -1;
  const long long want = (static_cast<long long>(B) * (rows[0] + rows[1]) * half + 255) / 256;
  return (int)launch_dependent(flux_rope_table_kernel, dim3(static_cast<unsigned>(want < 148LL * 16 ? want : 148LL * 16)), dim3(256), 0, (cudaStream_t)stream, a);
}

// out bf16 [B, dim]: cosines, then sines of t * factor * exp(-log_period * j / (dim / 2)).
extern "C" TYR_EXPORT int tyr_timestep_embedding(const float* t, void* out, int B, int dim, float factor, float log_period, void* stream) {
  if (B < 1 || dim < 2 || static_cast<long long>(B) * dim > (1LL << 30)) return -1;
  return (int)launch_dependent(timestep_embedding_kernel, dim3((B * dim + 255) / 256), dim3(256), 0, (cudaStream_t)stream, t, (__nv_bfloat16*)out, B, dim, factor, log_period);
}
