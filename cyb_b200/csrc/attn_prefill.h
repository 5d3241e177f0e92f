// Causal attention of prompt rows over the paged KV cache (attn_prefill.cu).
#pragma once
#include <cuda_bf16.h>

#include "qeng_internal.h"

struct qeng_prefill_attn {
  const __half* q16;       // [B*T][Hq][128]
  const int32_t* table;    // [B][max_pages]
  const int32_t* lens;     // [B*T] keys a row attends to (its position + 1)
  __nv_bfloat16* out;      // `planes` bf16 planes [B*T][ldo], `plane` elements apart
  long long ldo, plane;
  int planes;
  int B, T, Hq, Hkv, max_pages, pages;
  float scale, softcap;
  int window;
  int32_t* status;
};

// tensor map (128 bytes, 64-byte aligned) of a pool of `rows` rows of 128 f16
int32_t qeng_kv_map(qeng_ctx* ctx, void* pool, int64_t rows, void* map);
int32_t qeng_attn_prefill(qeng_ctx* ctx, const qeng_prefill_attn& p, const void* map, cudaStream_t stream);
// gemm_tc.cu: the driver's cuTensorMapEncodeTiled, or null
void* qeng_tensor_map_encoder();
