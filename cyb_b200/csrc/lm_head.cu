// LM head: logits[m][v] = softcap(sum_k norm(x)[m][k] * table[v][k]), bf16 table, up to 16 rows per launch, optionally
// with the greedy end of a decode step (sample, record, advance, embed the next token).
//
// HBM-bound: V * D * 2 bytes of table, read once whatever the number of rows.  The table is the A operand of tcgen05
// MMAs as it is; the activations are three bf16 planes, which hold a f32 exactly, as 48 columns of B.  A CTA owns `rpc`
// consecutive vocabulary rows (up to 256: two accumulators of 128 lanes), so that one round of CTAs covers a table of up
// to 256 rows per SM (37888 on 148) and several equal rounds a larger one;
// TMA brings 64-wide K chunks of them through a ring that keeps 200 KB in flight, filled before the kernel in front has
// ended.  Four warps write the activations of each chunk beside it, times the RMSNorm gain, and sum the squares as they
// go: the norm's factor is common to a row and multiplies its finished sums.  Tensor memory accumulates one chunk; the
// epilogue warps add the chunks up in registers with a compensated sum: what is left is the rounding inside a chunk.
// V = 32000, D = 4096: 45.8 us at 1 row, 48.0 us at 16 (5.5 TB/s).  One warp per vocabulary row with f32 FMAs, four rows a
// launch, took 54 and 590 us.
//
// Every wait is bounded; on expiry the kernel records status 4 and still frees its tensor memory.
#include <cuda.h>
#include <math.h>

#include "gemm_tc.cuh"

namespace {
using namespace qeng_tc;

constexpr int kM = 16, kCols = 3 * kM;   // rows per launch, their three planes
constexpr int kEpi = 8, kConv = 4, kThreadsL = (2 + kEpi + kConv) * 32;
constexpr int kMaxStagesL = 24;
constexpr int kTilePlane = 128 * kBK * 2;  // 128 table rows of a chunk
constexpr size_t kHeadSmem = kSmemBudget - 4096;  // dynamic; the static arrays take the rest
constexpr uint32_t kBBytes = kCols * 128u;

struct HeadParams {
  qeng_lm_tail t;
  int vec;                      // activations and gain 16-byte aligned
  int rpc, tiles, nk, nstages;  // vocabulary rows per tile, tiles, K chunks, ring stages
  float* part_val;              // [CTA][kM] best logit and its index
  int32_t* part_idx;
  int32_t* counter;
  int32_t* status;
};

__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int k, int row, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst), "l"(map),
               "r"(k), "r"(row), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void umma1(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b),
               "r"(idesc), "r"(acc)
               : "memory");
}
__device__ __forceinline__ void commit1(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool better(float v, int i, float bv, int bi) { return v > bv || (v == bv && i < bi); }
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(kEpi * 32) : "memory"); }

__global__ void __launch_bounds__(kThreadsL, 1) lm_head_kernel(const HeadParams p, const __grid_constant__ CUtensorMap wmap) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) uint64_t full[kMaxStagesL], empty[kMaxStagesL], acc_full[2], acc_empty[2], drained, ss_ready;
  __shared__ uint32_t tmem_slot;
  __shared__ float wv[kEpi][kM], ssq[kConv][kM];
  __shared__ int wi[kEpi][kM], tok[kM], s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t a_bytes = (uint32_t)p.rpc * 128u, stage = a_bytes + kBBytes;
  const int groups = p.rpc > 128 ? 2 : 1;

  if (tid == 0) {
    for (int s = 0; s < p.nstages; ++s) {
      mbar_init(smem_u32(full + s), 2);  // the producer and the warp that writes the activations
      mbar_init(smem_u32(empty + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(acc_full + b), 1);
      mbar_init(smem_u32(acc_empty + b), kEpi);
    }
    mbar_init(smem_u32(&drained), 1);
    mbar_init(smem_u32(&ss_ready), kConv);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;\n" ::"r"(smem_u32(&tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;
  bool failed = false;

  if (warp == 0) {
    // ===== producer of the table's chunks: they need nothing of the kernel before =================================
    if (elect_one()) {
      const int mine = (int)blockIdx.x < p.tiles ? (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0, total = mine * p.nk;
      for (int i = 0; i < total; ++i) {
        const int s = i % p.nstages;
        if (!mbar_wait(smem_u32(empty + s), ((uint32_t)(i / p.nstages) & 1u) ^ 1u)) { failed = true; break; }
        mbar_expect_tx(smem_u32(full + s), a_bytes);
        tma_2d(smem + (uint32_t)s * stage, &wmap, (i % p.nk) * kBK, ((int)blockIdx.x + i / p.nk * (int)gridDim.x) * p.rpc, smem_u32(full + s));
      }
      if (failed) atomicExch(p.status, 4);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ===== MMA issuer ==========================================================================================
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kCols >> 3) << 17) | (8u << 24);  // M = 128, N = 48
    int s = 0, n = 0;
    uint32_t ph = 0;
    for (int tile = blockIdx.x; tile < p.tiles && !failed; tile += gridDim.x)
      for (int kc = 0; kc < p.nk; ++kc) {
        const int buf = n & 1;
        if (!mbar_wait(smem_u32(acc_empty + buf), (((uint32_t)n >> 1) & 1u) ^ 1u)) failed = true;
        if (failed || !mbar_wait(smem_u32(full + s), ph)) failed = true;
        if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t a = __shfl_sync(0xffffffffu, smem + (uint32_t)s * stage, 0), d = __shfl_sync(0xffffffffu, tmem + (uint32_t)buf * 128u, 0);
        if (elect_one()) {
          const uint64_t ad = make_desc(a), bd = make_desc(a + a_bytes);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            const uint32_t acc = k > 0 ? 1u : 0u;
            umma1(d, ad + 2 * k, bd + 2 * k, idesc, acc);
            if (groups > 1) umma1(d + 64u, ad + (kTilePlane >> 4) + 2 * k, bd + 2 * k, idesc, acc);
          }
          commit1(smem_u32(empty + s));
          commit1(smem_u32(acc_full + buf));
        }
        __syncwarp();
        ++n;
        if (++s == p.nstages) { s = 0; ph ^= 1u; }
      }
    for (int b = 0; b < 2 && b < n; ++b) {  // the last accumulators have been read: nothing is in flight any more
      const int last = n - 1 - b;
      if (!failed && !mbar_wait(smem_u32(acc_empty + (last & 1)), ((uint32_t)last >> 1) & 1u)) failed = true;
    }
    if (failed) {
      if (elect_one()) commit1(smem_u32(&drained));
      __syncwarp();
      mbar_wait(smem_u32(&drained), 0);
      if (lane == 0) atomicExch(p.status, 4);
    }
  } else if (warp >= 2 + kEpi) {
    // ===== activations: warp w takes chunks w, w + 4, ...; a lane has 8 k of rows lane / 8, + 4, + 8, + 12 =========
    const qeng_lm_tail& t = p.t;
    const int w = warp - 2 - kEpi, c8 = lane & 7, r4 = lane >> 3;
    const int mine = (int)blockIdx.x < p.tiles ? (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0, total = mine * p.nk;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    float ss[kM / 4] = {};
    float4 x0[kM / 4], x1[kM / 4], g0 = make_float4(1.f, 1.f, 1.f, 1.f), g1 = g0;
    auto load8 = [&](const float* src, float4& a, float4& b) {
      if (p.vec) {
        a = reinterpret_cast<const float4*>(src)[0];
        b = reinterpret_cast<const float4*>(src)[1];
      } else {
        a = make_float4(src[0], src[1], src[2], src[3]);
        b = make_float4(src[4], src[5], src[6], src[7]);
      }
    };
    auto fetch = [&](int i) {  // zero beyond D, where the table's chunk is zero too
      const int k = (i % p.nk) * kBK + c8 * 8;
      const bool in = i < total && k < t.D;
      if (t.gamma != nullptr && in) load8(t.gamma + k, g0, g1);
#pragma unroll
      for (int j = 0; j < kM / 4; ++j) {
        const int m = r4 + 4 * j;
        x0[j] = x1[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in && m < t.M) load8(t.x + (size_t)m * t.D + k, x0[j], x1[j]);
      }
    };
    // The sums of squares are complete with the warp's last chunk of the first tile and are handed over right there: the
    // epilogue waits for them at the end of that tile, and until it goes on no ring stage of the second one is freed.
    bool published = false;
    auto publish = [&]() {
#pragma unroll
      for (int j = 0; j < kM / 4; ++j) {
        float v = ss[j];
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        if (c8 == 0) ssq[w][r4 + 4 * j] = v;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ss_ready));
      published = true;
    };
    if (w >= p.nk) publish();  // no chunk of the first tile is this warp's
    fetch(w);
    for (int i = w; i < total; i += kConv) {
      const int s = i % p.nstages;
      if (!failed && !mbar_wait(smem_u32(empty + s), ((uint32_t)(i / p.nstages) & 1u) ^ 1u)) failed = true;
      if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
      const uint32_t b = smem + (uint32_t)s * stage + a_bytes;
#pragma unroll
      for (int j = 0; j < kM / 4; ++j) {
        const int m = r4 + 4 * j;
        if (4 * j >= t.M) break;  // the columns of absent rows are never read
        const float v[8] = {x0[j].x, x0[j].y, x0[j].z, x0[j].w, x1[j].x, x1[j].y, x1[j].z, x1[j].w};
        const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        uint32_t o[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float a0 = v[2 * e] * g[2 * e], a1 = v[2 * e + 1] * g[2 * e + 1];
          if (i < p.nk) ss[j] = fmaf(v[2 * e], v[2 * e], fmaf(v[2 * e + 1], v[2 * e + 1], ss[j]));
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a0, a1);
            o[pl][e] = *reinterpret_cast<const uint32_t*>(&h);
            const float h0 = __uint_as_float(o[pl][e] << 16), h1 = __uint_as_float(o[pl][e] & 0xffff0000u);
            a0 = isinf(h0) ? 0.f : a0 - h0;  // an infinity is whole in the first plane
            a1 = isinf(h1) ? 0.f : a1 - h1;
          }
        }
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(b + (uint32_t)(pl * kM + m) * 128u + (uint32_t)((c8 ^ (m & 7)) << 4)),
                       "r"(o[pl][0]), "r"(o[pl][1]), "r"(o[pl][2]), "r"(o[pl][3])
                       : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(full + s));
      fetch(i + kConv);
      if (i < p.nk && i + kConv >= p.nk) publish();
    }
    if (!published) publish();
    if (failed && lane == 0) atomicExch(p.status, 4);
  } else {
    // ===== epilogue: lane = vocabulary row =======================================================================
    const qeng_lm_tail& t = p.t;
    const int ew = warp - 2, quad = warp & 3, grp = ew >> 2, row = grp * 128 + quad * 32 + lane, M = t.M;
    const int Vtot = t.Vtot > 0 ? t.Vtot : t.V;
    const size_t ldl = t.Vtot > 0 ? (size_t)t.ldl : (size_t)t.V;
    const bool finalise = t.next != nullptr || t.pairs != nullptr;
    float bestv[kM];
    int besti[kM];
#pragma unroll
    for (int m = 0; m < kM; ++m) { bestv[m] = -INFINITY; besti[m] = 0x7fffffff; }
    int n = 0;
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
      float acc[kM], low[kM];
#pragma unroll
      for (int m = 0; m < kM; ++m) acc[m] = low[m] = 0.f;
      for (int kc = 0; kc < p.nk; ++kc, ++n) {
        const int buf = n & 1;
        if (!failed && !mbar_wait(smem_u32(acc_full + buf), ((uint32_t)n >> 1) & 1u)) failed = true;
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (grp < groups) {
          const uint32_t src = tmem + (uint32_t)buf * 128u + (uint32_t)grp * 64u + ((uint32_t)(quad * 32) << 16);
          uint32_t v[kM], u[kM];
          tmem_ld16(src + 2 * kM, v);
          tmem_ld16(src + kM, u);
#pragma unroll
          for (int m = 0; m < kM; ++m) u[m] = __float_as_uint(__uint_as_float(u[m]) + __uint_as_float(v[m]));
          tmem_ld16(src, v);
#pragma unroll
          for (int m = 0; m < kM; ++m) {
            const float c = __uint_as_float(v[m]) + __uint_as_float(u[m]), sum = acc[m] + c;
            low[m] += c - (sum - acc[m]);
            acc[m] = sum;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(acc_empty + buf));
      }
#pragma unroll
      for (int m = 0; m < kM; ++m) acc[m] = isinf(acc[m]) ? acc[m] : acc[m] + low[m];  // an infinite sum has no remainder
      if (t.gamma != nullptr) {
        if (!failed && !mbar_wait(smem_u32(&ss_ready), 0)) failed = true;
#pragma unroll
        for (int m = 0; m < kM; ++m)
          if (m < M) acc[m] *= rsqrtf((ssq[0][m] + ssq[1][m] + ssq[2][m] + ssq[3][m]) / (float)t.D + t.eps);
      }
      const int v = tile * p.rpc + row;
      if (row < p.rpc && v < t.V && !failed) {
#pragma unroll
        for (int m = 0; m < kM; ++m) {
          if (m < M) {
            t.logits[(size_t)m * ldl + t.v0 + v] = t.softcap > 0.f ? t.softcap * tanhf(acc[m] / t.softcap) : acc[m];
            if (better(acc[m], t.v0 + v, bestv[m], besti[m])) { bestv[m] = acc[m]; besti[m] = t.v0 + v; }
          }
        }
      }
    }
    if (failed && lane == 0) atomicExch(p.status, 4);

    // ---- greedy finalisation: every CTA leaves its best per row, the one that arrives last picks (nobody waits) ----
    if (finalise) {
      const int et = tid - 64;  // 0 .. 255
#pragma unroll
      for (int m = 0; m < kM; ++m) {
        if (m < M) {
          float bv = bestv[m];
          int bi = besti[m];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
          }
          if (lane == 0) { wv[ew][m] = bv; wi[ew][m] = bi; }
        }
      }
      epi_sync();
      if (et < M) {
        float bv = wv[0][et];
        int bi = wi[0][et];
        for (int w = 1; w < kEpi; ++w)
          if (better(wv[w][et], wi[w][et], bv, bi)) { bv = wv[w][et]; bi = wi[w][et]; }
        __stcg(p.part_val + (size_t)blockIdx.x * kM + et, bv);
        __stcg(p.part_idx + (size_t)blockIdx.x * kM + et, bi);
      }
      __threadfence();
      epi_sync();
      if (et == 0) s_last = atomicAdd(p.counter, 1) == (int)gridDim.x - 1;
      epi_sync();
      if (s_last) {
        __threadfence();
        // 16 lanes per row m look at the CTAs' candidates
        const int m = et >> 4, l16 = et & 15;
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        if (m < M)
          for (int c = l16; c < (int)gridDim.x; c += 16) {
            const float v = __ldcg(p.part_val + (size_t)c * kM + m);
            const int i = __ldcg(p.part_idx + (size_t)c * kM + m);
            if (better(v, i, bv, bi)) { bv = v; bi = i; }
          }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (l16 == 0 && m < M) {
          if (t.pairs != nullptr) {  // a vocabulary shard: the ranks' (max, index) pairs meet in a later kernel
            t.pairs[2 * (t.pair_slot + m)] = bv;
            t.pairs[2 * (t.pair_slot + m) + 1] = (float)bi;  // exact: sharded vocabularies stay below 2^24
          } else {
            if ((unsigned)bi >= (unsigned)Vtot) { bi = 0; atomicExch(p.status, 3); }  // only if every logit was NaN
            tok[m] = bi;
            t.next[m] = bi;
            t.out_tokens[(size_t)(*t.step + 1) * M + m] = bi;
            t.pos[m] += 1;
            t.lens[m] += 1;
          }
        }
        epi_sync();
        if (et == 0) {
          if (t.pairs == nullptr) *t.step += 1;
          *p.counter = 0;  // ready for the next launch
        }
        if (t.pairs == nullptr) {
          const int nv = t.D / 8;
          for (int i = et; i < M * nv; i += kEpi * 32) {
            const int mm = i / nv, c = i - mm * nv;
            const uint4 w = reinterpret_cast<const uint4*>(t.emb + (size_t)tok[mm] * t.D)[c];
            float4* dst = reinterpret_cast<float4*>(t.xout + (size_t)mm * t.D) + 2 * c;
            dst[0] = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
            dst[1] = make_float4(__uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u), __uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u));
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  if (__syncthreads_or(failed)) grace();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;\n" ::"r"(tmem));
}

}  // namespace

int32_t qeng_lm_head_fused(qeng_ctx* ctx, const qeng_lm_tail& t, cudaStream_t stream) {
  if (t.M < 1 || t.M > kM) return qeng_fail(ctx, QENG_ERR_SHAPE, "lm_head: at most %d rows per launch", kM);
  if (t.V <= 0 || t.D <= 0 || t.D % 8 != 0) return qeng_fail(ctx, QENG_ERR_SHAPE, "lm_head: D must be a positive multiple of 8");
  if ((reinterpret_cast<uintptr_t>(t.table) & 15) != 0) return qeng_fail(ctx, QENG_ERR_ALIGN, "lm_head: table must be 16-byte aligned");
  HeadParams p;
  p.t = t;
  p.vec = ((reinterpret_cast<uintptr_t>(t.x) | reinterpret_cast<uintptr_t>(t.gamma)) & 15) == 0;
  // as few rounds of CTAs as 256 rows per CTA allow, the rows spread evenly over them
  const int rounds = (t.V + 256 * ctx->sm_count - 1) / (256 * ctx->sm_count);
  p.rpc = ((t.V + rounds * ctx->sm_count - 1) / (rounds * ctx->sm_count) + 7) / 8 * 8;
  if (p.rpc > 256) p.rpc = 256;
  p.tiles = (t.V + p.rpc - 1) / p.rpc;
  p.nk = (t.D + kBK - 1) / kBK;
  // an MMA reads 128 rows, also where fewer were loaded: the last stage is followed by what that may reach
  const size_t reach = (p.rpc > 128 ? 256 : 128) * 128, stage = (size_t)p.rpc * 128 + kBBytes, pad = reach > stage ? reach - stage : 0;
  p.nstages = (int)((kHeadSmem - 1024 - pad) / stage);
  if (p.nstages > kMaxStagesL) p.nstages = kMaxStagesL;
  p.part_val = ctx->tail_val; p.part_idx = ctx->tail_idx; p.counter = ctx->tail_cnt; p.status = ctx->status;
  auto enc = reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(qeng_tensor_map_encoder());
  CUtensorMap wmap;
  const cuuint32_t es[2] = {1, 1};
  const cuuint64_t wd[2] = {(cuuint64_t)t.D, (cuuint64_t)t.V}, st[1] = {(cuuint64_t)t.D * 2};
  const cuuint32_t wb[2] = {kBK, (cuuint32_t)p.rpc};
  if (!enc ||
      enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(t.table), wd, st, wb, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return qeng_fail(ctx, QENG_ERR_CUDA, "lm_head: tensor map rejected (V=%d, D=%d)", t.V, t.D);
  static bool configured_on[64] = {};  // the opt-in shared-memory size is set per device
  bool& configured = configured_on[ctx->device & 63];
  if (!configured) {
    QENG_CUDA(ctx, cudaFuncSetAttribute(lm_head_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHeadSmem));
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  cfg.stream = stream;
  cfg.gridDim = dim3((unsigned)(p.tiles < ctx->sm_count ? p.tiles : ctx->sm_count));
  cfg.blockDim = dim3(kThreadsL);
  cfg.dynamicSmemBytes = p.nstages * stage + pad + 1024;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, lm_head_kernel, p, wmap));
  return QENG_OK;
}
