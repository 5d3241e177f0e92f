// Causal attention of prompt rows (GQA) over the paged f16 KV cache.
//
// One CTA serves 64 MMA rows = 64 / group tokens x the query heads of one kv head, so a K / V tile fetched
// once is used by every head of the group (the decode kernel, called once per prompt row, fetched the whole
// context for every token: 16 GB per layer at 1800 tokens).  A producer warp brings pages into a ring of
// 32-token tiles, one TMA box of 8 KB per page, 128-byte swizzled so that ldmatrix reads are free of bank
// conflicts; four consumer warps own 16 rows each (mma.sync m16n8k16, f32 accumulation, online softmax).
// The probabilities enter the second product as two f16 terms, as in the decode kernel: no precision is
// lost there.  Three CTAs per SM.
//
// Least time: 24 MMAs of 2 cycles per 16 x 8 scores (8 for the scores, 16 for the values); 2 * 128 * 3 * heads * T^2 / 2
// operations for a prompt of T tokens = 73 us per layer at T = 1800 and 32 heads.  It takes 148 there (ncu; 212 with the
// CTAs in head order): the tensor pipe is busy 57 % of the cycles in which an SM has work (dependent steps of the softmax
// between the two products, 12 consumer warps per SM).
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>

#include <type_traits>

#include "attn_prefill.h"

namespace {

constexpr int kHD = 128, kNW = 4, kRows = 16 * kNW, kThreads = (kNW + 1) * 32;
constexpr int kTile = 32, kStages = 3, kPageBytes = 8192, kStageBytes = 2 * kPageBytes;
constexpr int kQBytes = kRows * kHD * 2;
constexpr size_t kSmem = kQBytes + kStages * kStageBytes + 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
// Bounded wait: gives up (false) two seconds after the first failed attempt.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
  unsigned long long t0;
  asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t0));
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t1;
    asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t1));
    if (t1 - t0 > 2000000000ull) return false;
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  return mbar_try_wait(bar, parity) || mbar_wait_slow(bar, parity);
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// byte offset of 16-byte chunk c (0..15) of row r in a tile of [2 halves][rows][128 B], 128-byte swizzled
__device__ __forceinline__ uint32_t chunk_at(int rows, int r, int c) {
  return (uint32_t)((c >> 3) * rows * 128 + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

__device__ __forceinline__ __half2 ldh2(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
  return *reinterpret_cast<__half2*>(&v);
}
// whether the values of a tile's keys up to kv1 hold an infinity or a NaN (asked by whole warps)
__device__ __forceinline__ bool tile_not_finite(uint32_t kv, int key0, int kv1, int lane) {
  uint32_t worst = 0;  // largest magnitude bits of the halves: an exponent of all ones has 0x7c00 and more
  if (key0 + lane < kv1) {  // lane = key
    const uint32_t row = kv + (uint32_t)(lane >> 4) * kPageBytes;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      uint4 v;
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                   : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                   : "r"(row + chunk_at(32, 16 + (lane & 15), c))
                   : "memory");
      worst = __vmaxu2(worst, __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu)));
    }
  }
  return __any_sync(0xffffffffu, (worst & 0xffffu) >= 0x7c00u || (worst >> 16) >= 0x7c00u);
}

__global__ void __launch_bounds__(kThreads, 3) attn_prefill_kernel(const qeng_prefill_attn p, const __grid_constant__ CUtensorMap kvmap) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t ring = base + kQBytes;
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages];
  __shared__ volatile int gave_up;  // a consumer stopped waiting: nobody waits for the producer's copies any more
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int grp = p.Hq / p.Hkv, tpt = kRows / grp;             // tokens per tile
  // long tiles first, of all heads and sequences together: head after head, the long tiles of the last heads started late
  // and an SM had work 65 % of the time
  const int hb = blockIdx.x % (unsigned)(p.Hkv * p.B), b = hb / p.Hkv, h = hb - b * p.Hkv;
  const int tt0 = (int)((gridDim.x - 1 - blockIdx.x) / (unsigned)(p.Hkv * p.B)) * tpt;
  const int ntok = min(tpt, p.T - tt0);

  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(full + s), 1);
      mbar_init(smem_u32(empty + s), kNW);
    }
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  // queries of this tile, zero rows where there is no token
  for (int i = tid; i < kRows * 16; i += kThreads) {
    const int r = i >> 4, c = i & 15, tok = r / grp;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (tok < ntok)
      v = *reinterpret_cast<const uint4*>(p.q16 + (((size_t)b * p.T + tt0 + tok) * p.Hq + (size_t)h * grp + (r - tok * grp)) * kHD + c * 8);
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(base + chunk_at(kRows, r, c)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
  }
  // keys any row of the tile attends to: [kv0, kv1)
  const int32_t* lens = p.lens + (size_t)b * p.T + tt0;
  int kv1 = 0, kv0 = 0x7fffffff, len_min = 0x7fffffff, win_max = 0;
  for (int i = lane; i < ntok; i += 32) {
    const int l = min(lens[i], p.max_pages * 16), w0 = p.window > 0 ? max(0, l - p.window) : 0;
    kv1 = max(kv1, l);
    len_min = min(len_min, l);
    kv0 = min(kv0, w0);
    win_max = max(win_max, w0);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    kv1 = max(kv1, __shfl_xor_sync(0xffffffffu, kv1, o));
    kv0 = min(kv0, __shfl_xor_sync(0xffffffffu, kv0, o));
    len_min = min(len_min, __shfl_xor_sync(0xffffffffu, len_min, o));
    win_max = max(win_max, __shfl_xor_sync(0xffffffffu, win_max, o));
  }
  const int t0 = kv0 / kTile, t1 = (kv1 + kTile - 1) / kTile;
  __syncthreads();

  bool failed = false;
  if (warp == kNW) {
    // ===== producer: two pages per tile; a page beyond the context repeats the last one (its keys are masked) ======
    const int last_page = (kv1 - 1) >> 4;
    int s = 0;
    uint32_t ph = 0;
    for (int kt = t0; kt < t1; ++kt) {
      const int pg = min(kt * 2 + (lane & 1), last_page);
      int pid = p.table[(size_t)b * p.max_pages + pg];
      if ((unsigned)pid >= (unsigned)p.pages) {  // malformed page table: record it, read a page that exists
        atomicExch(p.status, 1);
        pid = 0;
      }
      if (!failed && !mbar_wait(smem_u32(empty + s), ph ^ 1u)) failed = true;
      if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
      const uint32_t bar = smem_u32(full + s);
      if (lane == 0) mbar_expect_tx(bar, kStageBytes);
      __syncwarp();
      if (lane < 2) {
        const int row = (pid * p.Hkv + h) * 32;
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
                ring + (uint32_t)s * kStageBytes + (uint32_t)lane * kPageBytes),
            "l"(&kvmap), "r"(0), "r"(row), "r"(0), "r"(bar)
            : "memory");
      }
      if (++s == kStages) { s = 0; ph ^= 1u; }
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
    if (failed || gave_up) grace();
    return;
  }

  // ===== consumers: rows warp * 16 + g and + 8 =========================================================
  auto token_of = [&](int i) { return (warp * 16 + g + 8 * i) / grp; };  // worked out where needed: registers are short
  const float sc = p.scale * 1.4426950408889634f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float o[16][4];
#pragma unroll
  for (int j = 0; j < 16; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] = 0.f;

  // ldmatrix row of this lane: A (queries): rows 0..15, chunk lane/16; K: row lane%8, chunk lane/8; V: row lane%16, chunk lane/16
  const int qrow = warp * 16 + (lane & 15), qc = lane >> 4, krow = lane & 7, kc = lane >> 3, vrow = 16 + (lane & 15), vc = lane >> 4;
  // one tile of 32 keys; kEdge: not every row attends every key of it
  auto tile = [&](int kt, uint32_t kv, auto edge_tile) {
    constexpr bool kEdge = decltype(edge_tile)::value;
    int len[2], win[2];  // the keys that the lane's two rows attend: [win, len)
    if (kEdge) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        len[i] = token_of(i) < ntok ? min(lens[token_of(i)], p.max_pages * 16) : 0;
        win[i] = p.window > 0 ? max(0, len[i] - p.window) : 0;
      }
    }
    float sa[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) sa[n][0] = sa[n][1] = sa[n][2] = sa[n][3] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // 32 of the 128 dims
      uint32_t qa[2][4];
#pragma unroll
      for (int k = 0; k < 2; ++k) ldsm4(base + chunk_at(kRows, qrow, 4 * j + 2 * k + qc), qa[k]);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        uint32_t kb[4];
        ldsm4(kv + (uint32_t)(n >> 1) * kPageBytes + chunk_at(32, (n & 1) * 8 + krow, 4 * j + kc), kb);
        mma16816(sa[n], qa[0], kb[0], kb[1]);
        mma16816(sa[n], qa[1], kb[2], kb[3]);
      }
    }
    // scale (optionally soft-capped), log2 domain, mask
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float x = sa[n][c];
        if (p.softcap > 0.f) x = p.softcap * tanhf(x * p.scale / p.softcap) * 1.4426950408889634f;
        else x *= sc;
        if (kEdge) {
          const int key = kt * kTile + n * 8 + 2 * t + (c & 1), i = c >> 1;
          if (key >= len[i] || key < win[i]) x = -INFINITY;
        }
        sa[n][c] = x;
        mx[c >> 1] = fmaxf(mx[c >> 1], x);
      }
    float alpha[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      const float mn = fmaxf(m_run[i], mx[i]);
      const float ref = mn == -INFINITY ? 0.f : mn;  // nothing attended yet: all weights below are zero
      alpha[i] = exp2f(m_run[i] - ref);
      m_run[i] = mn;
      l_run[i] *= alpha[i];
      mx[i] = ref;
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        sa[n][c] = exp2f(sa[n][c] - mx[c >> 1]);
        l_run[c >> 1] += sa[n][c];
      }
    if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        o[j][0] *= alpha[0]; o[j][1] *= alpha[0];
        o[j][2] *= alpha[1]; o[j][3] *= alpha[1];
      }
    }
    // Where the rows attend different keys, a value that is not finite would reach rows that do not attend it (their weight
    // is zero, but zero times infinity is NaN): such a tile, which real caches do not hold, goes key by key.
    if (kEdge && tile_not_finite(kv, kt * kTile, kv1, lane)) {
#pragma unroll 1
      for (int k = 0; k < kTile; ++k) {
        const int n = k >> 3, c = k & 1, src = (lane & ~3) | ((k & 7) >> 1), key = kt * kTile + k;
        float w[2];  // weights of the lane's two rows for this key, from the lane of the quad that holds them
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float x = 0.f;
#pragma unroll
          for (int m = 0; m < 4; ++m)
            if (m == n) x = c ? sa[m][2 * i + 1] : sa[m][2 * i];
          w[i] = __shfl_sync(0xffffffffu, x, src);
        }
        const bool on0 = key < len[0] && key >= win[0], on1 = key < len[1] && key >= win[1];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float2 v = __half22float2(ldh2(kv + (uint32_t)(k >> 4) * kPageBytes + chunk_at(32, 16 + (k & 15), j) + (uint32_t)t * 4u));
          if (on0) { o[j][0] = fmaf(w[0], v.x, o[j][0]); o[j][1] = fmaf(w[0], v.y, o[j][1]); }
          if (on1) { o[j][2] = fmaf(w[1], v.x, o[j][2]); o[j][3] = fmaf(w[1], v.y, o[j][3]); }
        }
      }
    } else {
      const bool tail = kEdge && (kt + 1) * kTile > kv1;
#pragma unroll
      for (int pg = 0; pg < 2; ++pg) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // a0: keys 2t row g, a1: row g+8, a2 / a3: keys 2t + 8
          const float x = sa[2 * pg + (q >> 1)][2 * (q & 1)], y = sa[2 * pg + (q >> 1)][2 * (q & 1) + 1];
          hi[q] = pack_h2(x, y);
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi[q]));
          lo[q] = pack_h2(x - f.x, y - f.y);
        }
        // keys past the context: their weight is zero, but zero times whatever the page holds there may be NaN
        uint32_t keep[2] = {0xffffffffu, 0xffffffffu};
        if (tail) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int key = kt * kTile + pg * 16 + q * 8 + 2 * t;
            keep[q] = (key < kv1 ? 0xffffu : 0u) | (key + 1 < kv1 ? 0xffff0000u : 0u);
          }
        }
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
          uint32_t vb[4];
          ldsm4_t(kv + (uint32_t)pg * kPageBytes + chunk_at(32, vrow, c + vc), vb);
          if (tail) {
            vb[0] &= keep[0]; vb[1] &= keep[1];
            vb[2] &= keep[0]; vb[3] &= keep[1];
          }
          mma16816(o[c], hi, vb[0], vb[1]);
          mma16816(o[c + 1], hi, vb[2], vb[3]);
          mma16816(o[c], lo, vb[0], vb[1]);
          mma16816(o[c + 1], lo, vb[2], vb[3]);
        }
      }
    }
  };
  int s = 0;
  uint32_t ph = 0;
  for (int kt = t0; kt < t1; ++kt) {
    if (!failed && !mbar_wait(smem_u32(full + s), ph)) failed = true;
    const uint32_t kv = ring + (uint32_t)s * kStageBytes;
    if ((kt + 1) * kTile > len_min || kt * kTile < win_max || ntok < tpt) tile(kt, kv, std::true_type());
    else tile(kt, kv, std::false_type());
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(empty + s));
    if (++s == kStages) { s = 0; ph ^= 1u; }
  }
  if (failed) {
    gave_up = 1;
    if (lane == 0) atomicExch(p.status, 4);
    grace();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
    l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
    const int tok = token_of(i);
    if (tok >= ntok) continue;
    const float inv = l_run[i] > 0.f ? 1.f / l_run[i] : 0.f;
    const int head = h * grp + (warp * 16 + g + 8 * i) - tok * grp;
    const size_t at = ((size_t)b * p.T + tt0 + tok) * p.ldo + (size_t)head * kHD + 2 * t;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float x = o[j][2 * i] * inv, y = o[j][2 * i + 1] * inv;
      const __nv_bfloat162 hb = __floats2bfloat162_rn(x, y);
      *reinterpret_cast<__nv_bfloat162*>(p.out + at + j * 8) = hb;
      if (p.planes == 2)
        *reinterpret_cast<__nv_bfloat162*>(p.out + p.plane + at + j * 8) = __floats2bfloat162_rn(x - __low2float(hb), y - __high2float(hb));
    }
  }
}

}  // namespace

int32_t qeng_kv_map(qeng_ctx* ctx, void* pool, int64_t rows, void* map) {
  auto enc = qeng_tensor_map_encoder();
  // rows of 128 f16 as two halves of 64: a box of 32 rows x 2 halves is the K and V tile of one (page, kv head)
  const cuuint64_t dims[3] = {64, (cuuint64_t)rows, 2}, strides[2] = {256, 128};
  const cuuint32_t box[3] = {64, 32, 2}, es[3] = {1, 1, 1};
  if (!enc || reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(enc)(
                  reinterpret_cast<CUtensorMap*>(map), CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, pool, dims, strides, box, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return qeng_fail(ctx, QENG_ERR_CUDA, "attn_prefill: tensor map of the KV pool rejected");
  return QENG_OK;
}

int32_t qeng_attn_prefill(qeng_ctx* ctx, const qeng_prefill_attn& p, const void* map, cudaStream_t stream) {
  static bool configured_on[64] = {};  // the opt-in shared-memory size is set per device
  bool& configured = configured_on[ctx->device & 63];
  if (!configured) {
    QENG_CUDA(ctx, cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    configured = true;
  }
  const int tpt = kRows / (p.Hq / p.Hkv);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.T + tpt - 1) / tpt * p.Hkv * p.B));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, attn_prefill_kernel, p, *reinterpret_cast<const CUtensorMap*>(map)));
  return QENG_OK;
}
