// Causal attention of prompt rows (GQA) over the paged f16 KV cache, on the 5th-generation tensor cores.
//
// A tile is 128 MMA rows = 128 / group tokens x the query heads of one kv head, so a K / V page fetched once is used by every
// head of the group; a CTA works on two tiles of neighbouring tokens against the same keys, 64 at a time (four pages).  All
// operands but K and V live in tensor memory, 256 columns a tile: the queries (A operand of S = Q K^T), S, which the
// probabilities (A operand of O += P V, two f16 terms, so that no precision is lost there) overwrite, and O.  A page is one TMA
// box of 8 KB with a 128-byte swizzle; its K rows are a K-major B operand of 16 columns, its V rows an MN-major one of 128.
// Warps: 0-7 and 8-15 softmax of the two tiles, 16 MMA issue, 17 pages.  A lane of the softmax is a row and half of a tile's
// keys (no exchange between lanes; the two halves meet once a tile for the row's maximum).  The MMAs of one tile run while the
// other is in its softmax.  O is rescaled in tensor memory, only when a row's maximum has grown by more
// than 2^8 since it was last (the probabilities stay below 256, exact in two f16 terms as before).
//
// Least time: 64 keys of a tile are 32 MMAs of 16 columns (9.4 cycles each) and 8 of 128 (64): 815 cycles a tile, 37 K cycles
// for the 456 tiles of 1800 tokens, 32 query and 8 kv heads, on 148 SMs.  There a layer takes 68 us (ncu; 152 with mma.sync,
// whose pipe alone needs 73): what is left is the chain of a tile (scores, softmax, values, the hops between them), which two
// tiles a CTA hide by half.  128 tokens behind nothing 13.7 us (15.5), 16 x 45 tokens 13-16 (14.8): launch, first page, one
// chain.  A softmax of four warps a tile, a lane all 64 keys: 77 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>

#include "attn_prefill.h"

namespace {

constexpr int kHD = 128, kRows = 128, kTile = 64, kPages = kTile / 16, kStages = 3;
constexpr int kSoftWarps = 16, kMmaWarp = kSoftWarps, kLoadWarp = kMmaWarp + 1, kThreads = (kLoadWarp + 1) * 32;
constexpr int kKeys = kTile / 2;  // of a softmax warp
constexpr uint32_t kPageBytes = 8192, kStageBytes = kPages * kPageBytes;
constexpr uint32_t kScratch = kTile * kRows * 4;  // probabilities of a tile that goes key by key
constexpr size_t kSmem = kStages * kStageBytes + 2 * kScratch + 1024;
constexpr uint32_t kTileCols = 256, kO = 64, kS = 192;  // tensor-memory columns: queries at 0
constexpr float kGrow = 8.f;                            // log2 of how far a row's maximum may grow before O is rescaled

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
// the same for a converged warp, which learns the outcome by vote
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_b2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// 2^x, results below 2^-126 as zero
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
// shared-memory matrix descriptor, 128-byte swizzle.  K-major: 8-row groups `sbo` bytes apart (lbo unused); MN-major: groups of 64
// columns `lbo` apart, of 8 k `sbo` apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffff) >> 4);
  d |= (uint64_t)(lbo >> 4) << 16;
  d |= (uint64_t)(sbo >> 4) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  d |= (uint64_t)2 << 61;  // 128-byte swizzle
  return d;
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
#define R4(v, i) "=r"(v[i]), "=r"(v[i + 1]), "=r"(v[i + 2]), "=r"(v[i + 3])
#define R16(v, i) R4(v, i), R4(v, i + 4), R4(v, i + 8), R4(v, i + 12)
#define W4(v, i) "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3])
#define W16(v, i) W4(v, i), W4(v, i + 4), W4(v, i + 8), W4(v, i + 12)
// 32 columns of this warp's lanes (complete on return)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : R16(v, 0), R16(v, 16)
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31};\n" ::W16(v, 0), W16(v, 16), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n" ::W16(v, 0), "r"(taddr) : "memory");
}
#undef R4
#undef R16
#undef W4
#undef W16
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// address of 16-byte chunk c (0..15) of row r (16..31: V) of a page, [2 halves][32 rows][128 B], 128-byte swizzled
__device__ __forceinline__ uint32_t chunk_at(uint32_t page, int r, int c) {
  return page + (uint32_t)((c >> 3) * 4096 + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}

__global__ void __launch_bounds__(kThreads, 1) attn_prefill_kernel(const qeng_prefill_attn p, const int per_cta, const __grid_constant__ CUtensorMap kvmap) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) uint64_t kfull[kStages], kempty[kStages], sfull[2], pready[2], qready, odone, drained;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int skip_pv[2], not_finite[2][2][8];
  __shared__ float met[2][2][2][kRows];  // [turn][tile][half]: maxima of the rows, at the end their sums
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = p.Hq / p.Hkv, tpt = kRows / grp;  // tokens per tile
  // long tiles first, of all heads and sequences together
  const int hb = blockIdx.x % (unsigned)(p.Hkv * p.B), b = hb / p.Hkv, h = hb - b * p.Hkv;
  const int tt0 = (int)((gridDim.x - 1 - blockIdx.x) / (unsigned)(p.Hkv * p.B)) * tpt * per_cta;
  const int ntok = min(tpt * per_cta, p.T - tt0), tiles = (ntok + tpt - 1) / tpt;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(kfull + s), 1);
      mbar_init(smem_u32(kempty + s), 1);
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(smem_u32(sfull + x), 1);
      mbar_init(smem_u32(pready + x), kSoftWarps / 2);
      skip_pv[x] = 0;
    }
    mbar_init(smem_u32(&qready), kSoftWarps / 2 * tiles);
    mbar_init(smem_u32(&odone), 1);
    mbar_init(smem_u32(&drained), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    // Only now, with all of the SM's tensor memory in hand: the next kernel (the output projection) takes all of it, too, before it
    // waits for this one.  Where both fit on an SM (as compiled they do not, for registers and shared memory), one that came first
    // would hold what this CTA waits for.
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");

  // keys any row of the CTA attends to: [kv0, kv1); of this warp's own tile: what all its rows attend ends at len_min, begins at win_max
  const int32_t* lens = p.lens + (size_t)b * p.T + tt0;
  const int mine = warp < kSoftWarps ? warp >> 3 : 0;
  int kv1 = 0, kv0 = 0x7fffffff, len_min = 0x7fffffff, win_max = 0;
  for (int i = lane; i < ntok; i += 32) {
    const int l = min(lens[i], p.max_pages * 16), w0 = p.window > 0 ? max(0, l - p.window) : 0;
    kv1 = max(kv1, l);
    kv0 = min(kv0, w0);
    if (i / tpt == mine) {
      len_min = min(len_min, l);
      win_max = max(win_max, w0);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    kv1 = max(kv1, __shfl_xor_sync(0xffffffffu, kv1, o));
    kv0 = min(kv0, __shfl_xor_sync(0xffffffffu, kv0, o));
    len_min = min(len_min, __shfl_xor_sync(0xffffffffu, len_min, o));
    win_max = max(win_max, __shfl_xor_sync(0xffffffffu, win_max, o));
  }
  const int t0 = kv0 / kTile, t1 = (kv1 + kTile - 1) / kTile, n = max(t1 - t0, 0);
  bool failed = false;

  if (warp == kLoadWarp) {
    // ===== pages: four per stage; a page beyond the context repeats the last one (its keys are masked) ==============
    const int last_page = (kv1 - 1) >> 4;
    int s = 0;
    uint32_t ph = 1;
    for (int j = 0; j < n; ++j) {
      const int pg = min((t0 + j) * kPages + (lane & 3), last_page);
      int pid = p.table[(size_t)b * p.max_pages + pg];
      if ((unsigned)pid >= (unsigned)p.pages) {  // malformed page table: record it, read a page that exists
        atomicExch(p.status, 1);
        pid = 0;
      }
      if (!wait_warp(smem_u32(kempty + s), ph)) { failed = true; break; }
      const uint32_t bar = smem_u32(kfull + s);
      if (lane == 0) mbar_expect_tx(bar, kStageBytes);
      __syncwarp();
      if (lane < kPages) {
        const int row = (pid * p.Hkv + h) * 32;
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
                ring + (uint32_t)s * kStageBytes + (uint32_t)lane * kPageBytes),
            "l"(&kvmap), "r"(0), "r"(row), "r"(0), "r"(bar)
            : "memory");
      }
      if (++s == kStages) { s = 0; ph ^= 1u; }
    }
  } else if (warp == kMmaWarp) {
    // ===== MMA issue ================================================================================================
    const uint32_t base = __shfl_sync(0xffffffffu, ring, 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
    if (elect_one()) {
      // f16 x f16 -> f32, M = 128; S: N = 16, B K-major; O: N = 128, B MN-major
      constexpr uint32_t kIdescS = (1u << 4) | (2u << 17) | (8u << 24), kIdescO = (1u << 4) | (1u << 16) | (16u << 17) | (8u << 24);
      auto scores = [&](int x, int s) {
        const uint32_t q = tm + (uint32_t)x * kTileCols, page = base + (uint32_t)s * kStageBytes;
#pragma unroll
        for (int pg = 0; pg < kPages; ++pg) {
          const uint64_t kd = make_desc(page + pg * kPageBytes, 16, 1024);
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_f16(q + kS + 16 * pg, q + 8 * k, kd + (k >> 2) * (4096 >> 4) + (k & 3) * 2, kIdescS, k > 0);
        }
        umma_commit(smem_u32(sfull + x));
      };
      uint32_t begun = 0;  // bit x: tile x's O holds sums already
      auto values = [&](int x, int s) {
        const uint32_t t = tm + (uint32_t)x * kTileCols, page = base + (uint32_t)s * kStageBytes + 2048;
        if (!skip_pv[x]) {
#pragma unroll
          for (int pg = 0; pg < kPages; ++pg) {
            const uint64_t vd = make_desc(page + pg * kPageBytes, 4096, 1024);
            umma_f16(t + kO, t + kS + 8 * pg, vd, kIdescO, pg > 0 ? 1u : (begun >> x) & 1u);
            umma_f16(t + kO, t + kS + 32 + 8 * pg, vd, kIdescO, 1u);
          }
        }
        begun |= 1u << x;
      };
      failed = !mbar_wait(smem_u32(&qready), 0);
      if (!failed && n > 0) {
        failed = !mbar_wait(smem_u32(kfull), 0);
        fence_after();
        for (int x = 0; x < tiles && !failed; ++x) scores(x, 0);
      }
      int s = 0;
      uint32_t ph = 0;
      for (int j = 0; j < n && !failed; ++j) {
        const int s1 = s + 1 == kStages ? 0 : s + 1;
        const uint32_t ph1 = s1 == 0 ? ph ^ 1u : ph;
        for (int x = 0; x < tiles; ++x) {
          if (!mbar_wait(smem_u32(pready + x), (uint32_t)j & 1u)) { failed = true; break; }
          fence_after();
          values(x, s);
          if (x + 1 == tiles) umma_commit(smem_u32(j + 1 < n ? kempty + s : &odone));
          if (j + 1 < n) {
            if (x == 0 && !mbar_wait(smem_u32(kfull + s1), ph1)) { failed = true; break; }
            scores(x, s1);
          }
        }
        s = s1;
        ph = ph1;
      }
      if (failed) {  // what was issued still has to finish before tensor memory is freed
        umma_commit(smem_u32(&drained));
        mbar_wait(smem_u32(&drained), 0);
      }
    }
    failed = __any_sync(0xffffffffu, failed);
  } else if (mine < tiles) {
    // ===== softmax: this lane's row of tile `mine`, keys kKeys * half and on of each 64 ================================
    const int quad = warp & 3, half = (warp >> 2) & 1, row = quad * 32 + lane, tok = row / grp, at = mine * tpt + tok;
    const bool live = tok < tpt && at < ntok;
    const size_t token = (size_t)b * p.T + tt0 + at;
    const int head = h * grp + row - tok * grp;
    const uint32_t mem = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)mine * kTileCols;
    // the tile's warps.  What a warp writes to tensor memory behind it (probabilities over scores) another has read before it.
    auto meet = [&] {
      __syncwarp();
      fence_before();
      asm volatile("bar.sync %0, %1;\n" ::"r"(1 + mine), "n"(kSoftWarps / 2 * 32) : "memory");
      fence_after();
    };
    {
      uint32_t q[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (live) v = *reinterpret_cast<const uint4*>(p.q16 + (token * p.Hq + head) * kHD + half * 64 + i * 8);
        q[4 * i] = v.x; q[4 * i + 1] = v.y; q[4 * i + 2] = v.z; q[4 * i + 3] = v.w;
      }
      __syncwarp();
      tmem_st32(mem + 32 * half, q);
      st_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&qready));
    }
    // a row without a token attends everything, to nobody's use
    const int len = live ? min(lens[at], p.max_pages * 16) : 0x7fffffff, win = live && p.window > 0 ? max(0, len - p.window) : 0;
    const float sc = p.softcap > 0.f ? 1.f : p.scale * 1.4426950408889634f;
    float m_run = -INFINITY, l_run = 0.f;  // the row's maximum; the sum of this half's keys
    int slot = 0;
    uint32_t slot_ph = 0;
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      const int key0 = (t0 + j) * kTile;
      const bool edge = key0 + kTile > len_min || key0 < win_max;  // not every row attends every key (the same in all warps of the tile)
      if (!failed && !wait_warp(smem_u32(sfull + mine), (uint32_t)j & 1u)) failed = true;
      fence_after();
      float s[kKeys];
      tmem_ld32(mem + kS + kKeys * half, reinterpret_cast<uint32_t*>(s));
      if (p.softcap > 0.f) {
#pragma unroll
        for (int i = 0; i < kKeys; ++i) s[i] = p.softcap * tanhf(s[i] * p.scale / p.softcap) * 1.4426950408889634f;
      }
      if (edge) {
        const int end = len - key0 - kKeys * half, begin = win - key0 - kKeys * half;
#pragma unroll
        for (int i = 0; i < kKeys; ++i)
          if (i >= end || i < begin) s[i] = -INFINITY;
        // Where the rows attend different keys, a value that is not finite would reach rows that do not attend it (their weight
        // is zero, but zero times infinity is NaN): such a tile, which real caches do not hold, goes key by key.  Values of keys
        // past the context, which nobody attends, are cleared.  A warp looks after half the dims of one page.
        if (!failed && !wait_warp(smem_u32(kfull + slot), slot_ph)) failed = true;
        const uint32_t page = ring + (uint32_t)slot * kStageBytes + (uint32_t)quad * kPageBytes;
        const int r = 16 + (lane & 15), c0 = half * 8 + (lane >> 4) * 4;
        uint32_t worst = 0;  // largest magnitude bits of the halves: an exponent of all ones has 0x7c00 and more
        if (key0 + quad * 16 + (lane & 15) < kv1) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 v;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(chunk_at(page, r, c0 + c)) : "memory");
            worst = __vmaxu2(worst, __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu)));
          }
        } else if (mine == 0) {
#pragma unroll
          for (int c = 0; c < 4; ++c) asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};\n" ::"r"(chunk_at(page, r, c0 + c)), "r"(0u) : "memory");
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        }
        const bool any = __any_sync(0xffffffffu, (worst & 0xffffu) >= 0x7c00u || (worst >> 16) >= 0x7c00u);
        if (lane == 0) not_finite[mine][j & 1][warp & 7] = any;
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < kKeys; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], s[i]);
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      met[j & 1][mine][half][row] = mx;
      meet();
      mx = fmaxf(mx, met[j & 1][mine][half ^ 1][row]);
      bool bad = false;
      if (edge) {
#pragma unroll
        for (int i = 0; i < 8; ++i) bad = bad || not_finite[mine][j & 1][i];
      }
      // the reference of the row's exponentials moves when its maximum has left it far behind
      const bool moved = mx > m_run && (m_run == -INFINITY || (mx - m_run) * sc > kGrow);
      const float alpha = moved ? ex2((m_run - mx) * sc) : 1.f;
      if (moved) m_run = mx;
      l_run *= alpha;
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {  // this half's 64 dims
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t o[32];
          tmem_ld32(mem + kO + 64 * half + 32 * c, o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st32(mem + kO + 64 * half + 32 * c, o);
        }
      }
      const float off = m_run == -INFINITY ? 0.f : -m_run * sc;  // nothing attended yet: all weights are zero
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < kKeys; ++i) {
        s[i] = ex2(fmaf(s[i], sc, off));
        sum[i & 3] += s[i];
      }
      l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      if (!bad) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          hi[i] = pack_h2(s[2 * i], s[2 * i + 1]);
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi[i]));
          lo[i] = pack_h2(s[2 * i] - f.x, s[2 * i + 1] - f.y);
        }
        tmem_st16(mem + kS + 16 * half, hi);
        tmem_st16(mem + kS + 32 + 16 * half, lo);
      } else {
        const uint32_t w0 = ring + kStages * kStageBytes + (uint32_t)mine * kScratch + (uint32_t)row * 4u, pages = ring + (uint32_t)slot * kStageBytes;
#pragma unroll
        for (int i = 0; i < kKeys; ++i) asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(w0 + (uint32_t)(kKeys * half + i) * (kRows * 4)), "f"(s[i]) : "memory");
        meet();
        st_wait();
#pragma unroll 1
        for (int c = 2 * half; c < 2 * half + 2; ++c) {  // 32 of the 128 dims
          uint32_t o[32];
          if (j > 0) tmem_ld32(mem + kO + 32 * c, o);
          else
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
#pragma unroll 1
          for (int k = 0; k < kTile; ++k) {
            const bool on = key0 + k < len && key0 + k >= win;
            float w;
            asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(w) : "r"(w0 + (uint32_t)k * (kRows * 4)) : "memory");
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t v[4];
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                           : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                           : "r"(chunk_at(pages + (uint32_t)(k >> 4) * kPageBytes, 16 + (k & 15), 4 * c + q))
                           : "memory");
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v[i]));
                uint32_t* const d = o + 8 * q + 2 * i;
                if (on) {
                  d[0] = __float_as_uint(fmaf(w, f.x, __uint_as_float(d[0])));
                  d[1] = __float_as_uint(fmaf(w, f.y, __uint_as_float(d[1])));
                }
              }
            }
          }
          __syncwarp();
          tmem_st32(mem + kO + 32 * c, o);
        }
      }
      st_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) {
        if ((warp & 7) == 0) skip_pv[mine] = bad;
        mbar_arrive(smem_u32(pready + mine));
      }
      if (++slot == kStages) { slot = 0; slot_ph ^= 1u; }
    }
    if (n > 0 && !failed && !wait_warp(smem_u32(&odone), 0)) failed = true;
    fence_after();
    met[n & 1][mine][half][row] = l_run;
    meet();
    l_run += met[n & 1][mine][half ^ 1][row];
    // a row that attends nothing gives zeros (where no key is anybody's, O was never written); scores that are not finite give NaN
    const bool none = l_run == 0.f;
    const float inv = 1.f / l_run;
    __nv_bfloat16* const dst = p.out + token * p.ldo + (size_t)head * kHD + half * 64;
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      uint32_t o[32];
      __syncwarp();
      tmem_ld32(mem + kO + 64 * half + 32 * c, o);
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint32_t hw[4], lw[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float x = none ? 0.f : __uint_as_float(o[i + 2 * q]) * inv, y = none ? 0.f : __uint_as_float(o[i + 2 * q + 1]) * inv;
          hw[q] = pack_b2(x, y);
          const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hw[q]));
          lw[q] = pack_b2(x - f.x, y - f.y);
        }
        if (live) {
          *reinterpret_cast<uint4*>(dst + 32 * c + i) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
          if (p.planes == 2) *reinterpret_cast<uint4*>(dst + p.plane + 32 * c + i) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        }
      }
    }
  }
  if (failed && lane == 0) atomicExch(p.status, 4);
  fence_before();
  if (__syncthreads_or(failed)) grace();
  if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
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
  // Two tiles a CTA take turns on the tensor cores; with no more tiles than SMs each has one to itself.
  const int tpt = kRows / (p.Hq / p.Hkv), tiles = (p.T + tpt - 1) / tpt;
  const int per_cta = (int64_t)tiles * p.Hkv * p.B > ctx->sm_count ? 2 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((tiles + per_cta - 1) / per_cta * p.Hkv * p.B));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, attn_prefill_kernel, p, per_cta, *reinterpret_cast<const CUtensorMap*>(map)));
  return QENG_OK;
}
