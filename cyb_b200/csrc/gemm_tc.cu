// Quantised matmul of many activation rows on the 5th-generation tensor cores:
//   y[m][n] (f32) = sum_k x[m][k] * dequant(W)[n][k], f32 accumulation in tensor memory.
//
// The weights are the M side of the MMA, the activation rows ("tokens") its N side: an output tile is
// 256 weight rows x `bn` tokens, bn any multiple of 16 up to 256, so a token count that fits no tile
// wastes at most 15 columns of one, and the accumulator has one weight row per tensor-memory lane,
// which makes every store of the epilogue 128 contiguous bytes of a y row.
//
// A pair of CTAs (cluster of 2, tcgen05 cta_group::2) computes a tile: each CTA dequantises 128 of the
// weight rows and loads half of the tokens, so the activation tile crosses L2 -> shared memory once per
// pair and 64 k cost each SM 32 KB for 2 * 128 * bn * 64 MMA operations.  Roles (24 warps):
//   warp 0      issues tcgen05.mma (leader CTA, one thread); tcgen05.commit frees stages in both CTAs
//   warp 1      activation tiles: TMA boxes of 64 k x bn/2 tokens, 128-byte swizzle
//   warp 2      packed weights: one TMA box of 8 row tiles per stage and plane into a ring of its own,
//               which keeps tens of KB per SM in flight from HBM independently of the dequant warps
//   warp 3      tensor memory allocation
//   warps 4-7   epilogue (tcgen05.ld, one warp per lane quadrant), overlapped with the next tile: two
//               accumulators of 256 columns
//   warps 8-23  dequantisation: packed words -> bf16, stored in the swizzled K-major layout the MMA reads;
//               one warp per 16-row tile, two sets of 8 that take alternate stages
// A stage is KST chunks of 64 k: two where shared memory allows it (each role then pays its barrier
// round trips, some 300 cycles of dependent instructions, once per 128 k).
//
// Precision.  WP = 1 (prompt path of 4-bit blocks): weights and activations rounded to bf16, as before.
// WP = 2: a weight is the sum of two bf16 values (4-bit blocks: exact, (c-8)*s has 14 significant bits;
// 8-bit and K-quant blocks: 17 bits) and so are f32 / f16 activations (XP = 2; bf16 ones are exact as
// they are, XP = 1).  The products hi*hi + lo*hi + hi*lo accumulate in f32: relative error 2^-17 per
// operand, below the 15-bit block fixed point of the decode kernels.
//
// Work split: whole tiles round-robin over the CTA pairs while they fill waves; what is left over (all of
// it for a prompt chunk: 43 tiles of an 11008-row matrix cannot fill 74 pairs) is cut along K into equal
// shares (stream-K).  A pair leaves the partial sums of an unfinished tile in a workspace and a second
// kernel adds the parts in K order and runs the epilogue: the parts are a few MB in L2, which the whole
// chip sums in ~2 us, where one CTA per tile (the last to arrive) took 8 to 25 us.
//
// Every wait is bounded; on expiry the kernel records status 4, stops waiting and still frees its
// tensor memory before it returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <vector>

#include "gemm_tc.h"

namespace {

constexpr int kBK = 64;                  // k per chunk: one 128-byte swizzled row of bf16
constexpr int kDequantWarps = 8;         // per set
constexpr int kThreads = (8 + 2 * kDequantWarps) * 32;
constexpr int kAPlane = 128 * kBK * 2;   // 16 KB: this CTA's 128 weight rows of a chunk
constexpr int kMaxStages = 8, kMaxSlots = 12;
constexpr size_t kSmemBudget = 226 * 1024;

template <int FMT> struct Fmt;
template <> struct Fmt<QENG_FMT_Q4> { static constexpr int kW = 512, kS = 64; };
template <> struct Fmt<QENG_FMT_Q8> { static constexpr int kW = 1024, kS = 64; };
template <> struct Fmt<QENG_FMT_K4> { static constexpr int kW = 512, kS = 256; };
int chunk_w(int fmt) { return fmt == QENG_FMT_Q8 ? 1024 : 512; }
int chunk_s(int fmt) { return fmt == QENG_FMT_K4 ? 256 : 64; }
int slot_bytes_of(int fmt, int kst) { return kst * 8 * (chunk_w(fmt) + chunk_s(fmt)); }

struct TcParams {
  int nk;                    // stages of KST chunks along K
  int M, N;
  int bn, m_tiles, n_tiles;  // tokens per tile, token tiles, 256-row weight tiles
  int dp_tiles, sk_tiles;    // whole tiles (round-robin), tiles cut along K
  int nstages, nslots;       // rings: operand tiles, packed weights
  qeng_tc_epi e;
  int npairs;
  float* ws;                 // stream-K partials: [pair][2][CTA of the pair][bn][128]
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
// arrive on a barrier of either CTA of the pair (address from map_leader)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(1000u)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up (false) two seconds after the first failed attempt; a healthy wait ends
// in microseconds.  The clock is read once per 64 attempts.
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
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
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
__device__ __forceinline__ void sts128(uint32_t a, const uint32_t (&o)[4]) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
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
// the pair whose share holds unit u
__device__ __forceinline__ int pair_of_unit(long long U, int np, int u) {
  int q = (int)((long long)u * np / U);
  while (q + 1 < np && (int)(U * (q + 1) / np) <= u) ++q;
  while (q > 0 && (int)(U * q / np) > u) --q;
  return q;
}

// this lane's column (weight row `row` of its CTA) of pair q's partial of split tile r
__device__ __forceinline__ float* partial(const TcParams& p, int q, int r, uint32_t rank, int row) {
  const long long U = (long long)p.sk_tiles * p.nk;
  const int slot = (int)(U * q / p.npairs) / p.nk == r ? 0 : 1;  // the first tile of the pair's share, or a later one
  return p.ws + ((size_t)(q * 2 + slot) * 2 + rank) * p.bn * 128 + row;
}

// ---- dequantisation: one lane's words of one 32-block -> rows g and g+8, 8 consecutive k each ------------------
// The inner loop of the kernel: its rate is set by the integer pipe (half rate), so the 4-bit form spends two
// integer instructions per pair of weights (shift, AND-OR) and leaves the rest to the FMA pipe.
__device__ __forceinline__ __nv_bfloat162 bf2(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
__device__ __forceinline__ uint32_t u32(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }

// Codes in the low nibbles of bf16: 0x4300 | c is 128 + c; minus 136 gives c - 8 exactly.  The f16 scale is split
// into two bf16 terms (8 + 3 bits), so that the fma rounds (c-8)*s once, to the nearest bf16; the remainder is exact.
template <int WP>
__device__ __forceinline__ void dequant_q4(uint32_t w, float s, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  const uint32_t sb = __float_as_uint(s);
  const float rest = s - __uint_as_float(sb & 0xffff0000u);
  const __nv_bfloat162 s_hi = bf2(__byte_perm(sb, sb, 0x3232)), s_lo = bf2(__byte_perm(__float_as_uint(rest), __float_as_uint(rest), 0x3232));
  const __nv_bfloat162 off = bf2(0xc308c308u);  // -136
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // k = 2i and 2i + 1
    const __nv_bfloat162 c = __hadd2(bf2(((w >> (4 * i)) & 0x000f000fu) | 0x43004300u), off);
    const __nv_bfloat162 v = __hfma2(c, s_hi, __hmul2(c, s_lo));
    hi[i] = u32(v);
    if (WP == 2) lo[i] = u32(__hfma2(c, s_lo, __hfma2(c, s_hi, __hneg2(v))));
  }
}
// two f32 values -> bf16 pair and the bf16 pair of what the rounding left
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  hi = u32(h);
  lo = u32(__floats2bfloat162_rn(a - __low2float(h), b - __high2float(h)));
}
// block b (0 or 1) of the chunk at (wbase, sbase): hi/lo[0] row g, hi/lo[1] row g + 8
template <int FMT, int WP>
__device__ __forceinline__ void dequant_block(uint32_t wbase, uint32_t sbase, int lane, int b, uint32_t (&hi)[2][4], uint32_t (&lo)[2][4]) {
  const int g = lane >> 2;
  if (FMT == QENG_FMT_Q4) {
    const uint2 w = lds64(wbase + (uint32_t)(lane * 16 + b * 8));
    const uint32_t sp = lds32(sbase + (uint32_t)(g * 8 + b * 4));
    const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&sp));
    dequant_q4<WP>(w.x, sf.x, hi[0], lo[0]);
    dequant_q4<WP>(w.y, sf.y, hi[1], lo[1]);
  } else if (FMT == QENG_FMT_Q8) {
    const uint4 w = lds128(wbase + (uint32_t)(b * 512 + lane * 16));
    const uint32_t sp = lds32(sbase + (uint32_t)(g * 8 + b * 4));
    const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&sp));
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      // bytes of k = 0,4,1,5 and of k = 2,6,3,7; a signed byte xor 0x80 under the exponent of 2^23
      const uint32_t we = (r ? w.y : w.x) ^ 0x80808080u, wo = (r ? w.w : w.z) ^ 0x80808080u;
      const float s = r ? sf.y : sf.x;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t src = (i & 1) ? wo : we;
        const float a = __uint_as_float(__byte_perm(src, 0x4b000000u, 0x7440 + (i >> 1))) - 8388736.0f;
        const float c = __uint_as_float(__byte_perm(src, 0x4b000000u, 0x7442 + (i >> 1))) - 8388736.0f;
        split2(a * s, c * s, hi[r][i], lo[r][i]);
      }
    }
  } else {
    // per lane group: De(g), De(g+8), Do(g), Do(g+8) | Me(g), Me(g+8), Mo(g), Mo(g+8)
    const uint2 w = lds64(wbase + (uint32_t)(lane * 16 + b * 8));
    const uint2 d = lds64(sbase + (uint32_t)(g * 32 + b * 8)), m = lds64(sbase + (uint32_t)(g * 32 + 16 + b * 8));
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t wv = r ? w.y : w.x;
      const float D = __uint_as_float(r ? d.y : d.x), mn = __uint_as_float(r ? m.y : m.x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float a = __uint_as_float(0x4b000000u | ((wv >> (4 * i)) & 15u)) - 8388608.0f;
        const float c = __uint_as_float(0x4b000000u | ((wv >> (4 * i + 16)) & 15u)) - 8388608.0f;
        split2(fmaf(a, D, -mn), fmaf(c, D, -mn), hi[r][i], lo[r][i]);
      }
    }
  }
}

// ---- epilogue of up to 16 tokens of this lane's weight row -------------------------------------------------
// n = weight row of this lane (rows of a warp are 32 consecutive ones, so whole 16-row tiles); v[i] = sum of token m0 + i
__device__ __forceinline__ void st_planes(const qeng_tc_epi& e, size_t at, float f) {
  const __nv_bfloat16 h = __float2bfloat16_rn(f);
  e.yb[at] = h;
  if (e.yb_planes == 2) e.yb[at + e.yb_plane] = __float2bfloat16_rn(f - __bfloat162float(h));
}
__device__ __forceinline__ void finish16(const TcParams& p, int n, int m0, int cnt, const float (&v)[16], int lane) {
  const qeng_tc_epi& e = p.e;
  if (e.kind == QENG_EPI_STORE || e.kind == QENG_EPI_ACCUM) {
    if (n >= p.N) return;
    float* dst = e.y + (size_t)m0 * e.ldy + n;
    if (cnt >= 16) {
      if (e.kind == QENG_EPI_ACCUM) {
        float old[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) old[i] = dst[(size_t)i * e.ldy];
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[(size_t)i * e.ldy] = old[i] + v[i];
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[(size_t)i * e.ldy] = v[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (i < cnt) dst[(size_t)i * e.ldy] = e.kind == QENG_EPI_ACCUM ? dst[(size_t)i * e.ldy] + v[i] : v[i];
    }
    return;
  }
  // SWIGLU and QKV combine rows r and r + 8 of a 16-row tile: lanes with bit 3 clear take the even tokens, the others
  // the odd ones, so one exchange per token pair keeps every lane busy
  const int odd = (lane >> 3) & 1, r = lane & 7, tile = n >> 4;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 8);
    const float a = odd ? got : v[i], b = odd ? v[i + 1] : got;  // rows r and r + 8
    const int t = i + odd, m = m0 + t;
    if (t >= cnt || n >= p.N) continue;
    if (e.kind == QENG_EPI_SWIGLU) {
      const float f = a / (1.0f + __expf(-a)) * b;
      if (e.yb != nullptr) st_planes(e, (size_t)m * e.ldyb + (size_t)tile * 8 + r, f);
      else e.y[(size_t)m * e.ldy + (size_t)tile * 8 + r] = f;
    } else {
      const qeng_qkv_epi& q = e.qkv;
      const int head = tile >> 3, d = ((tile & 7) << 3) + r, ps = q.pos[m];
      if (ps < 0 || ps >= q.max_seq || (ps >> 4) >= q.max_pages) {
        atomicExch(p.status, 2);
        continue;
      }
      float lo = a, hi = b;
      if (head < q.Hq + q.Hkv) {
        const float c = q.cs[(size_t)ps * 128 + d], sn = q.cs[(size_t)ps * 128 + 64 + d];
        lo = a * c - b * sn;
        hi = b * c + a * sn;
      }
      __half* dst;
      if (head < q.Hq) {
        dst = q.q16 + ((size_t)m * q.Hq + head) * 128 + d;
      } else {
        const int pid = q.table[(size_t)(m / q.rows_per_seq) * q.max_pages + (ps >> 4)];
        if ((unsigned)pid >= (unsigned)q.pages) {
          atomicExch(p.status, 1);
          continue;
        }
        const int kh = head - q.Hq, isv = kh >= q.Hkv ? 1 : 0;
        dst = q.pool + (((size_t)pid * q.Hkv + (kh - isv * q.Hkv)) * 2 + isv) * (16 * 128) + (ps & 15) * 128 + d;
      }
      dst[0] = __float2half_rn(lo);
      dst[64] = __float2half_rn(hi);
    }
  }
}

template <int FMT, int WP, int XP, int KST>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                   const __grid_constant__ CUtensorMap smap) {
  constexpr int kW = Fmt<FMT>::kW, kS = Fmt<FMT>::kS;
  constexpr uint32_t kSlot = KST * 8 * (kW + kS);
  extern __shared__ unsigned char smem_raw[];
  // the swizzle pattern is a function of the address: tiles start on 1024-byte boundaries (the same offset in both CTAs)
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], wfull[kMaxSlots], wempty[kMaxSlots], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %cluster_ctarank;\n" : "=r"(rank));
  const int pair = blockIdx.x >> 1;
  const uint32_t b_plane = (uint32_t)(p.bn >> 1) * 128u;
  // stage: A [KST][WP] planes, then B [KST][XP] planes
  const uint32_t stage_bytes = KST * (WP * kAPlane + XP * b_plane);
  const uint32_t ring = smem + (uint32_t)p.nstages * stage_bytes;  // packed-weight slots

  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < p.nstages; ++s) {
      mbar_init(smem_u32(full + s), 1 + 2 * kDequantWarps);  // the leader's expect_tx, one set of dequant warps in each CTA
      mbar_init(smem_u32(empty + s), 1);
    }
    for (int s = 0; s < p.nslots; ++s) {
      mbar_init(smem_u32(wfull + s), 1);
      mbar_init(smem_u32(wempty + s), kDequantWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(acc_full + b), 1);
      mbar_init(smem_u32(acc_empty + b), 8);  // the epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;

  Segments segs(p, pair);
  Seg sg;
  bool failed = false;

  if (warp == 0) {
    // ===== MMA issuer =====================================================================
    if (rank == 0) {
      // f32 accumulate, bf16 x bf16, both K-major, N = bn, M = 256
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | (16u << 24);
      int s = 0, n = 0;
      uint32_t ph = 0;
      while (segs.next(p, sg)) {
        const int buf = n & 1;
        if (!failed && !mbar_wait(smem_u32(acc_empty + buf), (((uint32_t)n >> 1) & 1u) ^ 1u)) failed = true;
        const uint32_t d = tmem + (uint32_t)buf * 256u;
        for (int kt = sg.k0; kt < sg.k1; ++kt) {
          if (!failed && !mbar_wait(smem_u32(full + s), ph)) failed = true;
          __syncwarp();
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          if (elect_one()) {
            const uint32_t a = smem + (uint32_t)s * stage_bytes;
#pragma unroll
            for (int c = 0; c < KST; ++c) {
              const uint64_t ah = make_desc(a + c * WP * kAPlane), bh = make_desc(a + KST * WP * kAPlane + c * XP * b_plane);
#pragma unroll
              for (int k = 0; k < kBK / 16; ++k) {  // descriptors count 16-byte units: 2 per K step of 16
                umma_bf16(d, ah + 2 * k, bh + 2 * k, idesc, (kt > sg.k0 || c > 0 || k > 0) ? 1u : 0u);
                if (WP == 2) umma_bf16(d, ah + (kAPlane >> 4) + 2 * k, bh + 2 * k, idesc, 1u);
                if (XP == 2) umma_bf16(d, ah + 2 * k, bh + (b_plane >> 4) + 2 * k, idesc, 1u);
              }
            }
            umma_commit_pair(smem_u32(empty + s));
            if (kt + 1 == sg.k1) umma_commit_pair(smem_u32(acc_full + buf));
          }
          __syncwarp();
          if (++s == p.nstages) { s = 0; ph ^= 1u; }
        }
        ++n;
      }
      // the last accumulators have been read in both CTAs: nothing of this pair is in flight any more
      for (int b = 0; b < 2 && b < n; ++b) {
        const int last = n - 1 - b;
        if (!failed && !mbar_wait(smem_u32(acc_empty + (last & 1)), ((uint32_t)last >> 1) & 1u)) failed = true;
      }
      if (failed && lane == 0) atomicExch(p.status, 4);
    }
  } else if (warp == 1) {
    // ===== activation tiles ==================================================================
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    int s = 0;
    uint32_t ph = 0;
    while (!failed && segs.next(p, sg)) {
      int mt, nt;
      tile_pos(p, sg.tile, mt, nt);
      const int m0 = mt * p.bn + (int)rank * (p.bn >> 1);
      for (int kt = sg.k0; kt < sg.k1; ++kt) {
        if (!mbar_wait(smem_u32(empty + s), ph ^ 1u)) failed = true;
        if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(smem_u32(full + s), KST * XP * 2 * b_plane);
          const uint32_t b = smem + (uint32_t)s * stage_bytes + KST * WP * kAPlane, bar = map_leader(smem_u32(full + s));
#pragma unroll
          for (int c = 0; c < KST; ++c)
#pragma unroll
            for (int pl = 0; pl < XP; ++pl) tma_x(b + (uint32_t)(c * XP + pl) * b_plane, &xmap, (kt * KST + c) * kBK, m0, pl, bar);
        }
        __syncwarp();
        if (++s == p.nstages) { s = 0; ph ^= 1u; }
      }
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
  } else if (warp == 2) {
    // ===== packed weights ===================================================================
    int s = 0;
    uint32_t ph = 0;
    while (!failed && segs.next(p, sg)) {
      int mt, nt;
      tile_pos(p, sg.tile, mt, nt);
      for (int kt = sg.k0; kt < sg.k1; ++kt) {
        if (!mbar_wait(smem_u32(wempty + s), ph ^ 1u)) failed = true;
        if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
        if (elect_one()) {
          const uint32_t bar = smem_u32(wfull + s), dst = ring + (uint32_t)s * kSlot;
          mbar_expect_tx(bar, kSlot);
          tma_w(dst, &wmap, kt * KST, nt * 16 + (int)rank * 8, bar);
          tma_w(dst + KST * 8 * kW, &smap, kt * KST, nt * 16 + (int)rank * 8, bar);
        }
        __syncwarp();
        if (++s == p.nslots) { s = 0; ph ^= 1u; }
      }
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
  } else if (warp >= 8) {
    // ===== dequantisation: warp = one 16-row tile =================================================
    const int set = (warp - 8) >> 3, rt = (warp - 8) & 7, g = lane >> 2, t = lane & 3;
    // Lanes with odd g take the chunk's blocks in the other order: a quarter-warp then stores two rows into opposite
    // halves of the swizzled 128-byte line and touches every bank once.  dst[h]: row g, the h-th block this lane takes
    // (row g + 8 is 1024 bytes on: the swizzle depends on g alone).
    const int first = g & 1;
    uint32_t dst[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) dst[h] = smem + (uint32_t)((rt * 16 + g) * 128) + (uint32_t)((((h ^ first) * 4 + t) ^ g) << 4);
    const uint32_t wb0 = ring + (uint32_t)rt * (KST * kW), sb0 = ring + 8u * KST * kW + (uint32_t)rt * (KST * kS);
    int s = 0, ws = 0, turn = 0;  // turn: the set whose stage comes next
    uint32_t ph = 0, wph = 0;
    while (segs.next(p, sg)) {
      for (int kt = sg.k0; kt < sg.k1; ++kt) {
        if (turn == set) {
          if (!failed && !mbar_wait(smem_u32(wfull + ws), wph)) failed = true;
          const uint32_t wb = wb0 + (uint32_t)ws * kSlot, sb = sb0 + (uint32_t)ws * kSlot, so = (uint32_t)s * stage_bytes;
          uint32_t hi[2][2][4], lo[2][2][4];
#pragma unroll
          for (int h = 0; h < 2; ++h) dequant_block<FMT, WP>(wb, sb, lane, h ^ first, hi[h], lo[h]);
          if (!failed && !mbar_wait(smem_u32(empty + s), ph ^ 1u)) failed = true;
#pragma unroll
          for (int c = 0; c < KST; ++c) {
            if (c > 0) {
#pragma unroll
              for (int h = 0; h < 2; ++h)
                dequant_block<FMT, WP>(wb + (uint32_t)(c * kW), sb + (uint32_t)(c * kS), lane, h ^ first, hi[h], lo[h]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const uint32_t at = dst[h] + so + (uint32_t)(c * WP * kAPlane + r * 1024);
                sts128(at, hi[h][r]);
                if (WP == 2) sts128(at + kAPlane, lo[h][r]);
              }
          }
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            mbar_arrive_cluster(map_leader(smem_u32(full + s)));
            mbar_arrive(smem_u32(wempty + ws));
          }
        }
        turn ^= 1;
        if (++s == p.nstages) { s = 0; ph ^= 1u; }
        if (++ws == p.nslots) { ws = 0; wph ^= 1u; }
      }
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
  } else if (warp >= 4) {
    // ===== epilogue: warp = one quadrant of tensor-memory lanes =====================================
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int quad = warp & 3;
    int n = 0;
    while (segs.next(p, sg)) {
      int mt, nt;
      tile_pos(p, sg.tile, mt, nt);
      const int buf = n & 1, m0 = mt * p.bn, mcnt = min(p.bn, p.M - m0);
      const int row = quad * 32 + lane, wrow = nt * 256 + (int)rank * 128 + row;
      if (!failed && !mbar_wait(smem_u32(acc_full + buf), ((uint32_t)n >> 1) & 1u)) failed = true;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t tacc = tmem + (uint32_t)buf * 256u + ((uint32_t)(quad * 32) << 16);
      const bool whole = sg.k0 == 0 && sg.k1 == p.nk;
      float* mine = whole ? nullptr : partial(p, pair, sg.tile - p.dp_tiles, rank, row);
#pragma unroll 1
      for (int c0 = 0; c0 < mcnt; c0 += 16) {
        uint32_t v[16];
        tmem_ld16(tacc + (uint32_t)c0, v);
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
        if (failed) continue;
        if (whole) {
          finish16(p, wrow, m0 + c0, mcnt - c0, f, lane);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) __stcg(mine + (size_t)(c0 + i) * 128, f[i]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_leader(smem_u32(acc_empty + buf)));
      ++n;
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  cluster_sync();  // no CTA leaves while its peer may still signal it or read its shared memory
  if (warp == 3) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
}

// ---- tiles cut along K: the parts, added in K order, through the epilogue -----------------------------------
// Grid: (split tile, CTA of the pair) x 16 tokens; thread = weight row.
__global__ void __launch_bounds__(128) tc_reduce_kernel(const TcParams p) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int r = blockIdx.x >> 1, rank = blockIdx.x & 1, c0 = blockIdx.y * 16, row = threadIdx.x;
  const long long U = (long long)p.sk_tiles * p.nk;
  int mt, nt;
  tile_pos(p, p.dp_tiles + r, mt, nt);
  const int m0 = mt * p.bn, mcnt = min(p.bn, p.M - m0);
  const int q0 = pair_of_unit(U, p.npairs, r * p.nk), q1 = pair_of_unit(U, p.npairs, (r + 1) * p.nk - 1);
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  if (q0 == q1 || c0 >= mcnt) return;  // one pair had all of K: its epilogue is done
  float f[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = 0.f;
  for (int q = q0; q <= q1; ++q) {
    const float* src = partial(p, q, r, (uint32_t)rank, row) + (size_t)c0 * 128;
#pragma unroll
    for (int i = 0; i < 16; ++i) f[i] += __ldcg(src + (size_t)i * 128);
  }
  finish16(p, nt * 256 + rank * 128 + row, m0 + c0, mcnt - c0, f, row & 31);
}

// ---- activation rows -> one or two bf16 planes, optionally RMS-normalised on the way ----------------------
__global__ void __launch_bounds__(256) tc_prep_kernel(const void* __restrict__ x, int dtype, long long ldx, int K,
                                                      const float* __restrict__ gamma, float eps,
                                                      __nv_bfloat16* __restrict__ out, long long plane, int planes) {
  __shared__ float sh[8];
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int tid = threadIdx.x;
  const long long row = blockIdx.x;
  // K is a multiple of 32; a row of f32 may start at any 4-byte boundary
  const bool vec = dtype == QENG_F32 && ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ldx * 4)) & 15) == 0;
  auto load4 = [&](int k, float (&v)[4]) {
    if (vec) {
      const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + row * ldx + k);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const long long at = row * ldx + k + i;
        v[i] = dtype == QENG_F32 ? reinterpret_cast<const float*>(x)[at]
             : dtype == QENG_F16 ? __half2float(reinterpret_cast<const __half*>(x)[at])
                                 : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[at]);
      }
    }
  };
  float rs = 1.f;
  if (gamma != nullptr) {
    float ss = 0.f;
    for (int k = tid * 4; k < K; k += 1024) {
      float v[4];
      load4(k, v);
#pragma unroll
      for (int i = 0; i < 4; ++i) ss = fmaf(v[i], v[i], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) sh[tid >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) tot += sh[w];
    rs = rsqrtf(tot / (float)K + eps);
  }
  for (int k = tid * 4; k < K; k += 1024) {
    float v[4];
    load4(k, v);
    if (gamma != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = v[i] * rs * gamma[k + i];
    }
    uint2 hi, lo;
    split2(v[0], v[1], hi.x, lo.x);
    split2(v[2], v[3], hi.y, lo.y);
    *reinterpret_cast<uint2*>(out + row * K + k) = hi;
    if (planes == 2) *reinterpret_cast<uint2*>(out + plane + row * K + k) = lo;
  }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static const EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeFn>(f);
  }();
  return fn;
}

struct Plan {
  int kst, nk, bn, m_tiles, n_tiles, dp_tiles, sk_tiles, npairs, nstages, nslots;
  size_t smem, ws_floats;
};

// Tile width and split, by a cost model in cycles.  Per 64 k the MMAs take 2 * bn per product and the dequantisation a
// fixed time, whichever is longer; tiles cut along K pay for their partials' way through L2 and a second launch.
Plan make_plan(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int wp, int xp, bool may_split) {
  Plan best = {};
  double best_cost = 1e30;
  const int pairs = ctx->sm_count / 2, kst = wp == 1 ? 2 : 1, nk = (int)((w->nchunks + kst - 1) / kst);
  const int n_tiles = (int)((w->N + 255) / 256), products = wp + xp - 1;
  const double deq = kst * (w->fmt == QENG_FMT_Q4 ? (wp == 1 ? 330 : 450) : 700);
  const int lo = M <= 256 ? (int)((M + 15) / 16 * 16) : 128, hi = M <= 256 ? lo : 256;
  for (int bn = hi; bn >= lo; bn -= 16) {
    const int m_tiles = (int)((M + bn - 1) / bn), T = m_tiles * n_tiles;
    const double mma = 2.0 * kst * (bn < 32 ? 32 : bn) * products, stage = mma > deq ? mma : deq;
    const int waves = (T + pairs - 1) / pairs, rem = T % pairs;
    const double dp = waves * nk * stage + 25.0 * bn;
    const double sk = (T / pairs) * nk * stage + (double)rem * nk / pairs * stage + 50.0 * bn + 6000;
    // shares of at least two stages (with no whole tiles the number of pairs is reduced instead, below)
    const bool cut = may_split && rem != 0 && sk < dp && (T < pairs || (int64_t)rem * nk >= 2 * (int64_t)pairs);
    const double cost = cut ? sk : dp;
    if (cost < best_cost) {
      best_cost = cost;
      best.bn = bn; best.m_tiles = m_tiles; best.n_tiles = n_tiles;
      best.sk_tiles = cut ? rem : 0;
      best.dp_tiles = T - best.sk_tiles;
    }
  }
  best.kst = kst;
  best.nk = nk;
  best.npairs = best.sk_tiles > 0 ? pairs : (best.dp_tiles < pairs ? best.dp_tiles : pairs);
  if (best.sk_tiles > 0 && best.dp_tiles == 0) {
    const int64_t units = (int64_t)best.sk_tiles * nk;
    if (units / 2 < best.npairs) best.npairs = units / 2 > 0 ? (int)(units / 2) : 1;
  }
  // Operand stages first, but at least three slots of packed weights; what is left goes to the packed ring (few
  // tokens: the weights come from HBM and want tens of KB in flight, and then a stage leaves room for it).
  const size_t stage = (size_t)kst * (wp * kAPlane + xp * (best.bn / 2) * 128), slot = (size_t)slot_bytes_of(w->fmt, kst);
  const size_t room = kSmemBudget - 1024 - 1024;  // alignment, static shared memory
  best.nstages = (int)((room - 3 * slot) / stage);
  const int most = wp == 2 ? 4 : kMaxStages;
  if (best.nstages > most) best.nstages = most;
  best.nslots = (int)((room - best.nstages * stage) / slot);
  if (best.nslots > kMaxSlots) best.nslots = kMaxSlots;
  best.smem = best.nstages * stage + best.nslots * slot + 1024;
  best.ws_floats = best.sk_tiles > 0 ? (size_t)best.npairs * 4 * best.bn * 128 : 0;
  return best;
}

// tensor maps of the packed planes, boxes of kst chunks x 8 row tiles of 64-bit words; kept with the weight
bool weight_maps(const qeng_weight* w) {
  if (w->tc_maps_ready) return true;
  EncodeFn enc = encode_fn();
  for (int kst = 1; kst <= 2; ++kst)
    for (int plane = 0; plane < 2; ++plane) {
      const cuuint64_t words = (cuuint64_t)(plane == 0 ? chunk_w(w->fmt) : chunk_s(w->fmt)) / 8;
      const cuuint64_t dims[3] = {words, (cuuint64_t)w->nchunks, (cuuint64_t)w->ntiles};
      const cuuint64_t strides[2] = {words * 8, words * 8 * (cuuint64_t)w->nchunks};
      const cuuint32_t box[3] = {(cuuint32_t)words, (cuuint32_t)kst, 8}, es[3] = {1, 1, 1};
      void* base = plane == 0 ? reinterpret_cast<void*>(w->qs) : reinterpret_cast<void*>(w->sc);
      if (enc(reinterpret_cast<CUtensorMap*>(w->tc_maps[kst - 1][plane]), CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, base, dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    }
  w->tc_maps_ready = true;
  return true;
}

template <int FMT, int WP, int XP>
int32_t launch(qeng_ctx* ctx, const qeng_weight* w, const TcParams& p, const Plan& pl, const CUtensorMap& map, cudaStream_t stream) {
  constexpr int KST = WP == 1 ? 2 : 1;
  static bool configured_on[64] = {};  // the opt-in shared-memory size is set per device
  bool& configured = configured_on[ctx->device & 63];
  if (!configured) {
    QENG_CUDA(ctx, cudaFuncSetAttribute(gemm_tc_kernel<FMT, WP, XP, KST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pl.npairs));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  const CUtensorMap* wm = reinterpret_cast<const CUtensorMap*>(w->tc_maps[KST - 1][0]);
  const CUtensorMap* sm = reinterpret_cast<const CUtensorMap*>(w->tc_maps[KST - 1][1]);
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, gemm_tc_kernel<FMT, WP, XP, KST>, p, map, *wm, *sm));
  if (p.sk_tiles == 0) return QENG_OK;
  cfg.gridDim = dim3((unsigned)(2 * p.sk_tiles), (unsigned)(p.bn / 16));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, tc_reduce_kernel, p));
  return QENG_OK;
}

}  // namespace

void* qeng_tensor_map_encoder() { return reinterpret_cast<void*>(encode_fn()); }

int32_t qeng_tc_prep(qeng_ctx* ctx, const void* x, int32_t dtype, int64_t M, int64_t K, int64_t ldx, const float* gamma, float eps,
                     int planes, void* out, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)M);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, tc_prep_kernel, x, (int)dtype, (long long)ldx, (int)K, gamma, eps,
                                    reinterpret_cast<__nv_bfloat16*>(out), (long long)(M * K), planes));
  return QENG_OK;
}

int32_t qeng_gemm_tc(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, int wp, const qeng_tc_epi& epi, cudaStream_t stream) {
  const int xp = x.planes;
  if (w->fmt != QENG_FMT_Q4 && wp == 1) return qeng_fail(ctx, QENG_ERR_SHAPE, "gemm_tc: single bf16 weights are for 4-bit blocks only");
  if (wp == 1 && xp != 1) return qeng_fail(ctx, QENG_ERR_ARG, "gemm_tc: two activation planes need two weight planes");
  if ((reinterpret_cast<uintptr_t>(x.data) & 15) != 0 || (x.ld & 7) != 0)
    return qeng_fail(ctx, QENG_ERR_ALIGN, "gemm_q4 (prefill): activations must be 16-byte aligned with a leading dimension multiple of 8");
  qeng_scratch* sc = qeng_scratch_for(ctx, stream);
  Plan pl = make_plan(ctx, w, M, wp, xp, true);
  if (pl.sk_tiles > 0) {
    const int32_t rc = sc ? qeng_scratch_grow(ctx, &sc->part, pl.ws_floats * 4, stream) : QENG_ERR_STATE;
    if (rc != QENG_OK) pl = make_plan(ctx, w, M, wp, xp, false);  // no workspace inside this capture: whole tiles only
  }
  EncodeFn enc = encode_fn();
  if (!enc || !weight_maps(w)) return qeng_fail(ctx, QENG_ERR_CUDA, "gemm_tc: cuTensorMapEncodeTiled is not available or rejects the packed planes");
  CUtensorMap map;
  const cuuint64_t dims[3] = {(cuuint64_t)w->K, (cuuint64_t)M, (cuuint64_t)xp};
  const cuuint64_t strides[2] = {(cuuint64_t)x.ld * 2, (cuuint64_t)(xp > 1 ? x.plane : x.ld * M) * 2};
  const cuuint32_t box[3] = {kBK, (cuuint32_t)(pl.bn / 2), 1}, es[3] = {1, 1, 1};
  if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(x.data), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return qeng_fail(ctx, QENG_ERR_CUDA, "gemm_tc: tensor map rejected (M=%lld, K=%lld, ld=%lld)", (long long)M, (long long)w->K, (long long)x.ld);
  TcParams p;
  p.nk = pl.nk; p.M = (int)M; p.N = (int)w->N;
  p.bn = pl.bn; p.m_tiles = pl.m_tiles; p.n_tiles = pl.n_tiles; p.dp_tiles = pl.dp_tiles; p.sk_tiles = pl.sk_tiles;
  p.nstages = pl.nstages; p.nslots = pl.nslots; p.e = epi;
  p.ws = pl.sk_tiles > 0 ? reinterpret_cast<float*>(sc->part.ptr) : nullptr;
  p.npairs = pl.npairs;
  p.status = ctx->status;
  if (w->fmt == QENG_FMT_Q4) {
    if (wp == 1) return launch<QENG_FMT_Q4, 1, 1>(ctx, w, p, pl, map, stream);
    return xp == 1 ? launch<QENG_FMT_Q4, 2, 1>(ctx, w, p, pl, map, stream) : launch<QENG_FMT_Q4, 2, 2>(ctx, w, p, pl, map, stream);
  }
  if (w->fmt == QENG_FMT_Q8)
    return xp == 1 ? launch<QENG_FMT_Q8, 2, 1>(ctx, w, p, pl, map, stream) : launch<QENG_FMT_Q8, 2, 2>(ctx, w, p, pl, map, stream);
  return xp == 1 ? launch<QENG_FMT_K4, 2, 1>(ctx, w, p, pl, map, stream) : launch<QENG_FMT_K4, 2, 2>(ctx, w, p, pl, map, stream);
}

// y[M,N] = x . dequant(W)^T through the kernel above, activations in any type the entry point takes.
// wp = 1: operands rounded to bf16; wp = 2: two bf16 terms per weight and per f32 / f16 activation.
int32_t qeng_gemm_many_rows(qeng_ctx* ctx, const qeng_weight* w, const void* x, int32_t x_dtype, int64_t M, int64_t ldx, float* y, int64_t ldy,
                            int accumulate, int wp, cudaStream_t stream) {
  qeng_tc_epi e;
  e.kind = accumulate ? QENG_EPI_ACCUM : QENG_EPI_STORE;
  e.y = y;
  e.ldy = ldy;
  qeng_tc_x xx;
  const bool direct = x_dtype == QENG_BF16 && ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ldx * 2)) & 15) == 0;
  if (direct) {
    xx.data = x;
    xx.ld = ldx;
  } else {
    xx.planes = wp == 1 || x_dtype == QENG_BF16 ? 1 : 2;
    xx.ld = w->K;
    xx.plane = M * w->K;
    qeng_scratch* sc = qeng_scratch_for(ctx, stream);
    if (!sc) return qeng_fail(ctx, QENG_ERR_STATE, "gemm_q4: no activation scratch inside this stream capture (make one call of the shape before capturing)");
    int32_t rc = qeng_scratch_grow(ctx, &sc->planes, (size_t)xx.planes * M * w->K * 2, stream);
    if (rc == QENG_OK) rc = qeng_tc_prep(ctx, x, x_dtype, M, w->K, ldx, nullptr, 0.f, xx.planes, sc->planes.ptr, stream);
    if (rc != QENG_OK) return rc;
    xx.data = sc->planes.ptr;
  }
  return qeng_gemm_tc(ctx, w, xx, M, wp, e, stream);
}
