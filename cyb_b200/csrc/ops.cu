// Small operators of the decode loop: RMSNorm, RoPE, SwiGLU, residual add,
// embedding gather, greedy argmax.  All are HBM- or
// latency-bound elementwise / row-reduction kernels.
#include <math.h>

#include "qeng_internal.h"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float block_sum(float v, float* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < nw; ++w) tot += sh[w];
  return tot;
}

__global__ void rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ gamma, int D, float eps,
                               float* __restrict__ y) {
  __shared__ float sh[32];
  const float* xr = x + (size_t)blockIdx.x * D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) ss += xr[i] * xr[i];
  const float r = rsqrtf(block_sum(ss, sh) / (float)D + eps);
  for (int i = threadIdx.x; i < D; i += blockDim.x) y[(size_t)blockIdx.x * D + i] = xr[i] * r * gamma[i];
}

// standalone RoPE: angles in double so that no table is needed
__global__ void rope_kernel(float* x, const int32_t* pos, int H, int hd, float base) {
  const int m = blockIdx.x, half = hd / 2;
  for (int idx = threadIdx.x; idx < H * half; idx += blockDim.x) {
    const int h = idx / half, i = idx - h * half;
    const double ang = (double)pos[m] * pow((double)base, -2.0 * (double)i / (double)hd);
    double s, c;
    sincos(ang, &s, &c);
    float* p = x + ((size_t)m * H + h) * hd;
    const double a = p[i], b = p[i + half];
    p[i] = (float)(a * c - b * s);
    p[i + half] = (float)(b * c + a * s);
  }
}

__global__ void swiglu_kernel(const float* __restrict__ gate, const float* __restrict__ up, int64_t n,
                              float* __restrict__ y) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const float g = gate[i];
    y[i] = g / (1.0f + expf(-g)) * up[i];
  }
}

__global__ void add_kernel(const float* __restrict__ a, const float* __restrict__ b, int64_t n, float* __restrict__ y) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = a[i] + b[i];
}

__global__ void embed_kernel(const uint16_t* __restrict__ table, const int32_t* __restrict__ tokens, int D, int V,
                             float* __restrict__ x, int32_t* status) {
  const int m = blockIdx.x;
  int tok = tokens[m];
  if ((unsigned)tok >= (unsigned)V) {
    if (threadIdx.x == 0) atomicExch(status, 3);
    tok = 0;
  }
  for (int i = threadIdx.x; i < D; i += blockDim.x)
    x[(size_t)m * D + i] = __uint_as_float((uint32_t)table[(size_t)tok * D + i] << 16);
}

__global__ void argmax_kernel(const float* __restrict__ logits, int V, int32_t* __restrict__ idx) {
  __shared__ float bv[32];
  __shared__ int bi[32];
  const float* row = logits + (size_t)blockIdx.x * V;
  float best = -INFINITY;
  int besti = 0x7fffffff;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float v = row[i];
    if (v > best || (v == best && i < besti)) { best = v; besti = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
    if (ov > best || (ov == best && oi < besti)) { best = ov; besti = oi; }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { bv[warp] = best; bi[warp] = besti; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (bv[w] > best || (bv[w] == best && bi[w] < besti)) { best = bv[w]; besti = bi[w]; }
    idx[blockIdx.x] = besti == 0x7fffffff ? 0 : besti;
  }
}

}  // namespace

extern "C" {

int32_t qeng_rmsnorm(qeng_ctx* ctx, const float* x, const float* gamma, int64_t M, int64_t D, float eps, float* y,
                     void* stream) {
  if (!ctx || !x || !gamma || !y) return qeng_fail(ctx, QENG_ERR_ARG, "rmsnorm: null argument");
  if (M <= 0 || D <= 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "rmsnorm: empty shape");
  QENG_ENTER(ctx);
  rmsnorm_kernel<<<(unsigned)M, 256, 0, (cudaStream_t)stream>>>(x, gamma, (int)D, eps, y);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

int32_t qeng_rope(qeng_ctx* ctx, float* x, const int32_t* pos, int64_t M, int64_t H, int64_t hd, float base,
                  void* stream) {
  if (!ctx || !x || !pos) return qeng_fail(ctx, QENG_ERR_ARG, "rope: null argument");
  if (M <= 0 || H <= 0 || hd <= 0 || hd % 2) return qeng_fail(ctx, QENG_ERR_SHAPE, "rope: bad shape");
  QENG_ENTER(ctx);
  rope_kernel<<<(unsigned)M, 256, 0, (cudaStream_t)stream>>>(x, pos, (int)H, (int)hd, base);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

int32_t qeng_swiglu(qeng_ctx* ctx, const float* gate, const float* up, int64_t n, float* y, void* stream) {
  if (!ctx || !gate || !up || !y) return qeng_fail(ctx, QENG_ERR_ARG, "swiglu: null argument");
  if (n <= 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "swiglu: empty shape");
  QENG_ENTER(ctx);
  swiglu_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(gate, up, n, y);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

int32_t qeng_add(qeng_ctx* ctx, const float* a, const float* b, int64_t n, float* y, void* stream) {
  if (!ctx || !a || !b || !y) return qeng_fail(ctx, QENG_ERR_ARG, "add: null argument");
  if (n <= 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "add: empty shape");
  QENG_ENTER(ctx);
  add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(a, b, n, y);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

int32_t qeng_embed(qeng_ctx* ctx, const uint16_t* table_bf16, const int32_t* tokens, int64_t M, int64_t D, int64_t V,
                   float* x, void* stream) {
  if (!ctx || !table_bf16 || !tokens || !x) return qeng_fail(ctx, QENG_ERR_ARG, "embed: null argument");
  if (M <= 0 || D <= 0 || V <= 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "embed: empty shape");
  QENG_ENTER(ctx);
  embed_kernel<<<(unsigned)M, 256, 0, (cudaStream_t)stream>>>(table_bf16, tokens, (int)D, (int)V, x, ctx->status);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

int32_t qeng_lm_head(qeng_ctx* ctx, const uint16_t* table_bf16, const float* x, int64_t M, int64_t D, int64_t V,
                                float* logits, void* stream) {
  if (!ctx || !table_bf16 || !x || !logits) return qeng_fail(ctx, QENG_ERR_ARG, "lm_head: null argument");
  if (M <= 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "lm_head: empty shape");
  QENG_ENTER(ctx);
  for (int64_t m0 = 0; m0 < M; m0 += kHeadRows) {
    qeng_lm_tail t;
    t.table = table_bf16; t.x = x + m0 * D; t.M = (int)(M - m0 < kHeadRows ? M - m0 : kHeadRows); t.D = (int)D; t.V = (int)V;
    t.logits = logits + m0 * V;
    int32_t rc = qeng_lm_head_fused(ctx, t, (cudaStream_t)stream);
    if (rc != QENG_OK) return rc;
  }
  return QENG_OK;
}

int32_t qeng_argmax(qeng_ctx* ctx, const float* logits, int64_t M, int64_t V, int32_t* idx, void* stream) {
  if (!ctx || !logits || !idx) return qeng_fail(ctx, QENG_ERR_ARG, "argmax: null argument");
  if (M <= 0 || V <= 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "argmax: empty shape");
  QENG_ENTER(ctx);
  argmax_kernel<<<(unsigned)M, 1024, 0, (cudaStream_t)stream>>>(logits, (int)V, idx);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

}  // extern "C"
