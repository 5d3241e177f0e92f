// Building blocks of the matmuls of many rows: barriers, TMA, tcgen05, the work split over CTA pairs
// (gemm_tc.cu), and the epilogues (also gemm_rows.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "gemm_tc.h"

namespace qeng_tc {

constexpr int kBK = 64;                  // k per chunk: one 128-byte swizzled row of bf16
constexpr int kACols = kBK / 2;          // tensor-memory columns of one plane of a chunk of weights
constexpr int kMaxStages = 8, kMaxSlots = 12;
constexpr size_t kSmemBudget = 226 * 1024;

template <int FMT> struct Fmt;
template <> struct Fmt<QENG_FMT_Q4> { static constexpr int kW = 512, kS = 64; };
template <> struct Fmt<QENG_FMT_Q8> { static constexpr int kW = 1024, kS = 64; };
template <> struct Fmt<QENG_FMT_K4> { static constexpr int kW = 512, kS = 256; };
inline int chunk_w(int fmt) { return fmt == QENG_FMT_Q8 ? 1024 : 512; }
inline int chunk_s(int fmt) { return fmt == QENG_FMT_K4 ? 256 : 64; }
inline int slot_bytes_of(int fmt, int kst) { return kst * 8 * (chunk_w(fmt) + chunk_s(fmt)); }

struct TcParams {
  int nk;                    // stages of KST chunks along K
  int M, N;
  int bn, m_tiles, n_tiles;  // tokens per tile, token tiles, 256-row weight tiles
  int dp_tiles, sk_tiles;    // whole tiles (round-robin), tiles cut along K
  int nstages, nslots;       // rings: operands (weights in tensor memory, activations in shared memory), packed weights
  int nacc, acc_cols;        // accumulators (1 or 2), tensor-memory columns of each
  qeng_tc_epi e;
  int npairs;
  float* ws;                 // stream-K partials: [pair][2][CTA of the pair][bn / 4][128][4]
  int32_t* status;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_leader(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// Arrive on a barrier of either CTA of the pair (address from map_leader); whoever waits for it uses mbar_wait_cluster.
// Without the scope the arrival would be one among this CTA's threads alone.  It is relaxed: what is handed over is tensor
// memory, written or read to the end (wait::st, wait::ld) and fenced (before_thread_sync) ahead of it.  A release would also
// hold it back until the CTA's stores to global memory have reached L2 (8192 rows bf16 over 4096 x 11008: 578 -> 779 us).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
// CLUSTER: what the other CTA of the pair did before its arrival is seen, too
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (CLUSTER)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
// Bounded wait: gives up (false) two seconds after the first failed attempt; a healthy wait ends
// in microseconds.  The clock is read once per 64 attempts.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
  unsigned long long t0;
  asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t0));
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
    unsigned long long t1;
    asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t1));
    if (t1 - t0 > 2000000000ull) return false;
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  return mbar_try_wait(bar, parity) || mbar_wait_slow(bar, parity);
}
// The same for a converged warp and a barrier on which the other CTA arrives; all lanes learn the outcome by vote, so that
// what follows stays warp-uniform.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_try_wait<true>(bar, parity)) || __all_sync(0xffffffffu, mbar_wait_slow<true>(bar, parity));
}
// one box of a packed plane: `box` chunks x 8 row tiles (beyond the matrix: zeros)
__device__ __forceinline__ void tma_w(uint32_t dst, const CUtensorMap* map, int chunk, int tile, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
      "l"(map), "r"(0), "r"(chunk), "r"(tile), "r"(bar)
      : "memory");
}
// one box of the activation planes into this CTA's shared memory; the bytes are counted on the leader's barrier
__device__ __forceinline__ void tma_x(uint32_t dst, const CUtensorMap* map, int k, int m, int plane, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
      "l"(map), "r"(k), "r"(m), "r"(plane), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// 64-bit shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffff) >> 4);  // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset
  d |= (uint64_t)1 << 46;                   // descriptor version of this architecture
  d |= (uint64_t)2 << 61;                   // 128-byte swizzle
  return d;
}
// A from tensor memory (each CTA's 128 rows in its own), B from both CTAs' shared memory
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
// 16 lanes x 32 columns; a lane's registers 4i, 4i + 1: row g, columns 8i + 2t and the next; 4i + 2, 4i + 3: row g + 8
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n" ::"r"(v[0]), "r"(v[1]),
      "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
      "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr)
      : "memory");
}
// arrives at the barrier at this offset in both CTAs once the MMAs issued so far have finished
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
// one lane of a converged warp: lets the operands of the instructions it issues stay warp-uniform
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}

// ---- the sequence of (tile, K range) segments of one CTA pair; every role walks the same one ----------
struct Seg {
  int tile, k0, k1;
};
struct Segments {
  int next_dp, npairs, u, u1;
  __device__ Segments(const TcParams& p, int pair) : next_dp(pair), npairs(p.npairs) {
    const long long U = (long long)p.sk_tiles * p.nk;
    u = (int)(U * pair / npairs);
    u1 = (int)(U * (pair + 1) / npairs);
  }
  __device__ int stages(const TcParams& p) const {  // of all segments still to come
    return (next_dp < p.dp_tiles ? (p.dp_tiles - next_dp + npairs - 1) / npairs * p.nk : 0) + (u1 - u);
  }
  __device__ bool next(const TcParams& p, Seg& s) {
    if (next_dp < p.dp_tiles) {
      s.tile = next_dp;
      s.k0 = 0;
      s.k1 = p.nk;
      next_dp += npairs;
      return true;
    }
    if (u >= u1) return false;
    const int r = u / p.nk;
    s.tile = p.dp_tiles + r;
    s.k0 = u - r * p.nk;
    s.k1 = min(p.nk, s.k0 + (u1 - u));
    u += s.k1 - s.k0;
    return true;
  }
};
// Tiles in groups of 8 token tiles, weight tiles inside a group: a wave of pairs then works on few distinct
// activation tiles and few weight tiles at once, and both are read from HBM once per wave.
__device__ __forceinline__ void tile_pos(const TcParams& p, int tile, int& mt, int& nt) {
  const int grp = 8 * p.n_tiles, gi = tile / grp, first = gi * 8, rows = min(8, p.m_tiles - first);
  const int r = tile - gi * grp;
  mt = first + r % rows;
  nt = r / rows;
}
// The pair whose share holds unit u: the last one whose first unit, floor(U * q / np), is not beyond it.  (No divisions of 64
// bits: with them the sums of 16 tokens cost less than finding their parts.)
__device__ __forceinline__ int pair_of_unit(long long U, int np, int u) {
  const long long past = (long long)(u + 1) * np;  // floor(U * q / np) <= u where U * q is less
  int q = (int)((double)u * np / (double)U);
  while (q + 1 < np && U * (q + 1) < past) ++q;
  while (q > 0 && U * q >= past) --q;
  return q;
}

// weight row `row` of its CTA in pair q's partial of split tile r, of which q has a share: four tokens together, the next four
// 512 floats on (one 16-byte access per lane for four of 4 bytes: 192 rows f32 over 4096 x 4096 31.2 -> 30.3 us)
__device__ __forceinline__ float* partial(const TcParams& p, int q, int r, uint32_t rank, int row) {
  const long long U = (long long)p.sk_tiles * p.nk;
  const int slot = U * q >= (long long)r * p.nk * p.npairs ? 0 : 1;  // the first tile of the pair's share, or a later one
  return p.ws + ((size_t)(q * 2 + slot) * 2 + rank) * p.bn * 128 + row * 4;
}

__device__ __forceinline__ __nv_bfloat162 bf2(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }


// ---- epilogue of up to NT (8 or 16) tokens of this lane's weight row -------------------------------------------------
// n = weight row of this lane (rows of a warp are 32 consecutive ones, so whole 16-row tiles); v[i] = sum of token m0 + i
template <int NT>
__device__ __forceinline__ void finish(const qeng_tc_epi& e, int N, int32_t* status, int n, int m0, int cnt, const float (&v)[NT], int lane) {
  if (e.kind == QENG_EPI_STORE || e.kind == QENG_EPI_ACCUM) {
    if (n >= N) return;
    float* dst = e.y + (size_t)m0 * e.ldy + n;
    if (cnt >= NT) {
      if (e.kind == QENG_EPI_ACCUM) {
        float old[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) old[i] = dst[(size_t)i * e.ldy];
#pragma unroll
        for (int i = 0; i < NT; ++i) dst[(size_t)i * e.ldy] = old[i] + v[i];
      } else {
#pragma unroll
        for (int i = 0; i < NT; ++i) dst[(size_t)i * e.ldy] = v[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < NT; ++i)
        if (i < cnt) dst[(size_t)i * e.ldy] = e.kind == QENG_EPI_ACCUM ? dst[(size_t)i * e.ldy] + v[i] : v[i];
    }
    return;
  }
  // SWIGLU and QKV combine rows r and r + 8 of a 16-row tile: lanes with bit 3 clear take the even tokens, the others
  // the odd ones, so one exchange per token pair keeps every lane busy
  const int odd = (lane >> 3) & 1, r = lane & 7, tile = n >> 4;
  constexpr int kP = NT / 2;
  float lo[kP], hi[kP];  // rows r and r + 8 of token 2 i + odd
#pragma unroll
  for (int i = 0; i < kP; ++i) {
    const float got = __shfl_xor_sync(0xffffffffu, odd ? v[2 * i] : v[2 * i + 1], 8);
    lo[i] = odd ? got : v[2 * i];
    hi[i] = odd ? v[2 * i + 1] : got;
  }
  if (e.kind == QENG_EPI_SWIGLU) {
    // each step for all tokens before the next: token after token, with a branch for each, the chain of exchange, exponential,
    // division and stores took 4500 cycles per 16 tokens, more than the matmul of the next tile hides
    float den[kP];
#pragma unroll
    for (int i = 0; i < kP; ++i) den[i] = 1.0f + __expf(-lo[i]);
#pragma unroll
    for (int i = 0; i < kP; ++i) lo[i] = lo[i] / den[i] * hi[i];
    if (n >= N) return;
    if (e.yb != nullptr) {
      __nv_bfloat16* dst = e.yb + (size_t)(m0 + odd) * e.ldyb + (size_t)tile * 8 + r;
#pragma unroll
      for (int i = 0; i < kP; ++i) {
        const __nv_bfloat16 h = __float2bfloat16_rn(lo[i]);
        if (2 * i + odd < cnt) {
          dst[(size_t)(2 * i) * e.ldyb] = h;
          if (e.yb_planes == 2) dst[(size_t)(2 * i) * e.ldyb + e.yb_plane] = __float2bfloat16_rn(lo[i] - __bfloat162float(h));
        }
      }
    } else {
      float* dst = e.y + (size_t)(m0 + odd) * e.ldy + (size_t)tile * 8 + r;
#pragma unroll
      for (int i = 0; i < kP; ++i)
        if (2 * i + odd < cnt) dst[(size_t)(2 * i) * e.ldy] = lo[i];
    }
    return;
  }
  // QKV: the loads of all tokens (positions, then angles, then pages) are issued together: one after the other they were
  // three trips to L2 per token pair, and the epilogue of 1800 rows took twice as long as its matmul.
  const qeng_qkv_epi& q = e.qkv;
  const int head = tile >> 3, d = ((tile & 7) << 3) + r;
  int ps[kP];
#pragma unroll
  for (int i = 0; i < kP; ++i) ps[i] = 2 * i + odd < cnt && n < N ? q.pos[m0 + 2 * i + odd] : 0;
  bool ok[kP];
#pragma unroll
  for (int i = 0; i < kP; ++i) {
    ok[i] = 2 * i + odd < cnt && n < N;
    if (ok[i] && (ps[i] < 0 || ps[i] >= q.max_seq || (ps[i] >> 4) >= q.max_pages)) {
      atomicExch(status, 2);
      ok[i] = false;
    }
    if (!ok[i]) ps[i] = 0;
  }
  if (head < q.Hq + q.Hkv) {
    float c[kP], sn[kP];
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      c[i] = __ldg(q.cs + (size_t)ps[i] * 128 + d);
      sn[i] = __ldg(q.cs + (size_t)ps[i] * 128 + 64 + d);
    }
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      const float a = lo[i], b = hi[i];
      lo[i] = a * c[i] - b * sn[i];
      hi[i] = b * c[i] + a * sn[i];
    }
  }
  if (head < q.Hq) {
    __half* dst = q.q16 + ((size_t)(m0 + odd) * q.Hq + head) * 128 + d;
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      if (!ok[i]) continue;
      dst[(size_t)(2 * i) * q.Hq * 128] = __float2half_rn(lo[i]);
      dst[(size_t)(2 * i) * q.Hq * 128 + 64] = __float2half_rn(hi[i]);
    }
    return;
  }
  const int kh = head - q.Hq, isv = kh >= q.Hkv ? 1 : 0;
  int pid[kP];
#pragma unroll
  for (int i = 0; i < kP; ++i)
    pid[i] = ok[i] ? q.table[(size_t)((m0 + 2 * i + odd) / q.rows_per_seq) * q.max_pages + (ps[i] >> 4)] : 0;
#pragma unroll
  for (int i = 0; i < kP; ++i) {
    if (!ok[i]) continue;
    if ((unsigned)pid[i] >= (unsigned)q.pages) {
      atomicExch(status, 1);
      continue;
    }
    __half* dst = q.pool + (((size_t)pid[i] * q.Hkv + (kh - isv * q.Hkv)) * 2 + isv) * (16 * 128) + (ps[i] & 15) * 128 + d;
    dst[0] = __float2half_rn(lo[i]);
    dst[64] = __float2half_rn(hi[i]);
  }
}

struct Plan {
  int kst, nk, bn, m_tiles, n_tiles, dp_tiles, sk_tiles, npairs, nstages, nslots, nacc, acc_cols;
  bool pairs;    // whole tiles by drain_pairs
  int box_rows;  // rows of an activation box
  size_t smem, ws_floats;
};
// gemm_tc.cu: kernel parameters and the tensor map of the activations for a plan; QENG_ERR_STATE when the plan cuts
// tiles along K and there is no memory for the workspace
int32_t prepare(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, const qeng_tc_epi& epi, qeng_scratch* sc,
                const Plan* pl, TcParams* p, CUtensorMap* map);
// sums the partials of the tiles cut along K
int32_t reduce(qeng_ctx* ctx, const TcParams& p, cudaStream_t stream);

}  // namespace qeng_tc
