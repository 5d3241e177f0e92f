// Tensor-core matmul of many activation rows (gemm_tc.cu) and the per-stream scratch it works in.
#pragma once
#include <cuda_bf16.h>

#include "qeng_internal.h"

// What happens to the finished sums of a tile.
struct qeng_tc_epi {
  int kind = QENG_EPI_STORE;  // STORE, ACCUM (y += ...), SWIGLU (N/2 columns out), QKV (rotary, q16 and KV pages)
  float* y = nullptr;
  long long ldy = 0;
  // SWIGLU only: the result as one or two bf16 planes (the operand of the next matmul) instead of f32
  __nv_bfloat16* yb = nullptr;
  long long ldyb = 0, yb_plane = 0;
  int yb_planes = 1;
  qeng_qkv_epi qkv = {};
};

// Activations as bf16 planes: value = plane 0 (+ plane 1), rows `ld` apart, planes `plane` elements apart.
struct qeng_tc_x {
  const void* data = nullptr;
  long long ld = 0, plane = 0;
  int planes = 1;
};

// wp = 1: weights rounded to bf16 (4-bit blocks only); wp = 2: weights as two bf16 terms.  sc: the stream's working memory
// where the caller has looked it up already.
int32_t qeng_gemm_tc(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, int wp, const qeng_tc_epi& epi, cudaStream_t stream,
                     qeng_scratch* sc = nullptr);
// the same for rows of any type; wp = 1: operands rounded to bf16; wp = 2: two bf16 terms per weight and f32 / f16 activation
int32_t qeng_gemm_many_rows(qeng_ctx* ctx, const qeng_weight* w, const void* x, int32_t x_dtype, int64_t M, int64_t ldx, qeng_tc_epi e, int wp,
                            cudaStream_t stream);
// the driver's cuTensorMapEncodeTiled, or null
void* qeng_tensor_map_encoder();
// rows of x (any type), RMS-normalised if gamma is given -> `planes` bf16 planes [M][K]; with `sums` also their sums per
// 32-block, [planes][M][blocks, rounded up to an even number]
int32_t qeng_tc_prep(qeng_ctx* ctx, const void* x, int32_t dtype, int64_t M, int64_t K, int64_t ldx, const float* gamma, float eps,
                     int planes, void* out, float* sums, cudaStream_t stream);

// gemm_rows.cu: a few rows (all formats) at the precision of wp = 2; planes: 1 for bf16 rows, else 2
bool qeng_gemm_rows_fits(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int planes);
// whether the kernel can take them at all, faster or not
bool qeng_gemm_rows_planned(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int planes);
int32_t qeng_gemm_rows_reserve(qeng_ctx* ctx, const qeng_weight* w, int64_t M, cudaStream_t stream);
// rows of any type, converted by the matmul itself
int32_t qeng_gemm_rows_raw(qeng_ctx* ctx, const qeng_weight* w, const void* x, int32_t dtype, int64_t M, int64_t ldx, const qeng_tc_epi& epi, cudaStream_t stream);
// f32 rows, converted (and normalised, if gamma is given) by a kernel of its own: what the layers of a decoder take, where that kernel
// starts before the one in front of it has ended (sixteen rows converted and normalised by the matmul itself: 3270 us a step, so 2680)
int32_t qeng_gemm_rows_prep(qeng_ctx* ctx, const qeng_weight* w, const float* x, int64_t M, int64_t ldx, const float* gamma, float eps,
                            const qeng_tc_epi& epi, cudaStream_t stream);
// rows that are bf16 planes already (not K-quant blocks, which need the planes' block sums)
int32_t qeng_gemm_rows(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, const qeng_tc_epi& epi, cudaStream_t stream);
