// Quantised matmul of many activation rows on the 5th-generation tensor cores:
//   y[m][n] (f32) = sum_k x[m][k] * dequant(W)[n][k], f32 accumulation in tensor memory.
//
// The weights are the M side of the MMA, the activation rows ("tokens") its N side: an output tile is
// 256 weight rows x `bn` tokens, bn any multiple of 16 up to 256 (a plan may leave more than 15 columns of
// the last tile empty: 257 rows over 11008 x 4096 are two tiles of 144), and the accumulator has one weight
// row per tensor-memory lane, which makes every store of the epilogue 128 contiguous bytes of a y row.
//
// A pair of CTAs (cluster of 2, tcgen05 cta_group::2) computes a tile: each CTA dequantises 128 of the
// weight rows into its tensor memory, which is where the MMAs take their A operand from, and loads half of
// the tokens into shared memory, so the activation tile crosses L2 -> shared memory once per pair.
// Roles (24 warps):
//   warp 0      leader CTA: issues tcgen05.mma (one thread); tcgen05.commit frees stages in both CTAs.
//               Other CTA: passes its dequant warps' arrivals on to the leader, one per stage
//   warp 1      activation tiles: TMA boxes of 64 k x bn/2 tokens, 128-byte swizzle
//   warp 2      packed weights: one TMA box of 8 row tiles per stage and plane into a ring of its own,
//               which keeps tens of KB per SM in flight from HBM independently of the dequant warps
//   warp 3      tensor memory allocation
//   warps 4-7   epilogue (tcgen05.ld, one warp per lane quadrant), overlapped with the next tile where
//               there are two accumulators
//   warps 8-23  dequantisation: packed words -> bf16 -> tensor memory; one warp per 16-row tile, two sets
//               of 8 that take alternate stages; with one accumulator that is added to y also its epilogue
// A stage is two chunks of 64 k or (two weight terms, as the plan finds better) one, with one barrier each way: a hop between
// the roles costs 100 to 200 cycles of dependent instructions, and with one barrier per chunk the hops of a stage took longer
// than its MMAs.
// The weights used to pass through shared memory, which then carried 1.3 times what it can in the time of the MMAs; cycles per
// 128 k and one term, shared / tensor memory: 1460 / 1024 at 256 columns (the MMAs: 1024), 1240 / 800 to 880 at 160 (640); two
// terms, 112 columns: 2640 / 1340 (1344).  With it went the second accumulator of more than 160 columns (96 to 192 in two terms).
// Calls with weights through shared memory / now: 777 rows f32 over 11008 x 4096 86 / 68 us, 101 rows 36.0 / 30.8, 240 rows
// 57.0 / 57.2, over 4096 x 4096 32.6 / 27.8; 8192 rows bf16 over 4096 x 11008 627 / 549, 4096 rows added to y over 22016 x 4096
// 652 / 652; a prompt of 1800 tokens 33.2 / 24.4 ms.
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
#include <algorithm>

#include "gemm_tc.cuh"

namespace {
using namespace qeng_tc;

constexpr int kDequantWarps = 8, kSets = 2;
constexpr int kHelpers = kSets * kDequantWarps;
constexpr int kThreads = (8 + kHelpers) * 32;

// ---- dequantisation: one lane's words of one 32-block -> rows g and g+8, 8 consecutive k each ------------------
// The inner loop of the kernel: its rate is set by the integer pipe (half rate), so the 4-bit form spends two
// integer instructions per pair of weights (shift, AND-OR) and leaves the rest to the FMA pipe.
// Codes in the low nibbles of bf16: 0x4300 | c is 128 + c; minus 136 gives c - 8 exactly.  The f16 scale is split
// into two bf16 terms (8 + 3 bits), so that the fma rounds (c-8)*s once, to the nearest bf16; the remainder is exact.
struct Scale2 {
  __nv_bfloat162 hi, lo;
};
__device__ __forceinline__ Scale2 split_scale(float s) {
  const uint32_t sb = __float_as_uint(s);
  const uint32_t rest = __float_as_uint(s - __uint_as_float(sb & 0xffff0000u));
  return {bf2(__byte_perm(sb, sb, 0x3232)), bf2(__byte_perm(rest, rest, 0x3232))};
}
// (a & b) | c in one instruction, the constants in registers
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;\n" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ uint32_t in_register(uint32_t v) {
  uint32_t r;
  asm volatile("mov.u32 %0, %1;\n" : "=r"(r) : "r"(v));
  return r;
}
// the pair of codes in bits 0..3 and 16..19
template <int WP>
__device__ __forceinline__ void pair_q4(uint32_t w, const Scale2& s, uint32_t mask, uint32_t base, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 c = __hadd2(bf2(and_or(w, mask, base)), bf2(0xc308c308u));  // -136
  const __nv_bfloat162 v = __hfma2(c, s.hi, __hmul2(c, s.lo));
  hi = u32(v);
  if (WP == 2) lo = u32(__hfma2(c, s.lo, __hfma2(c, s.hi, __hneg2(v))));
}
// two f32 values -> bf16 pair and the bf16 pair of what the rounding left
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  hi = u32(h);
  lo = u32(__floats2bfloat162_rn(a - __low2float(h), b - __high2float(h)));
}
// One lane's share of a chunk, in the layout of tmem_st16: quad i = k 16i + 4t .. 16i + 4t + 3 of rows g and g + 8.
// Packed lane t' of a block holds k = 8t' .. 8t' + 7, so quad i of a block (i = 0, 1) is half t & 1 of the words of packed
// lane 2i + t / 2: neighbouring lanes read the same 16 bytes, each uses its half.
template <int FMT>
struct Words {   // 4-bit and K-quant blocks
  uint4 q0, q1;  // quad 0 / 1: row g and g + 8 of the first block, of the second
  uint4 d, m;    // K-quant: De(g), De(g+8), Do(g), Do(g+8) | Me(g), Me(g+8), Mo(g), Mo(g+8); 4-bit: d.x, d.y = f16 pairs
  __device__ __forceinline__ void load(uint32_t wbase, uint32_t sbase, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t w0 = wbase + (uint32_t)((g * 4 + (t >> 1)) * 16);
    q0 = lds128(w0);
    q1 = lds128(w0 + 32);
    if (FMT == QENG_FMT_K4) {
      d = lds128(sbase + (uint32_t)(g * 32));
      m = lds128(sbase + (uint32_t)(g * 32 + 16));
    } else {
      const uint2 s = lds64(sbase + (uint32_t)(g * 8));
      d = make_uint4(s.x, s.y, 0u, 0u);
      m = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  template <int WP>
  __device__ __forceinline__ void dequant(int lane, uint32_t mask, uint32_t base, uint32_t (&hi)[16], uint32_t (&lo)[16]) const {
    const uint32_t sh = 8u * (lane & 1);
    const uint32_t ws[2][2][2] = {{{q0.x, q1.x}, {q0.y, q1.y}}, {{q0.z, q1.z}, {q0.w, q1.w}}};  // [block][row][quad]
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const uint32_t s2 = b ? d.y : d.x;
      const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&s2));
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const Scale2 s = split_scale(r ? sf.y : sf.x);
        const float D = __uint_as_float(b ? (r ? d.w : d.z) : (r ? d.y : d.x)), mn = __uint_as_float(b ? (r ? m.w : m.z) : (r ? m.y : m.x));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t w = ws[b][r][i] >> sh;
          const int at = (b * 2 + i) * 4 + r * 2;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (FMT == QENG_FMT_Q4) {
              pair_q4<WP>(w >> (4 * j), s, mask, base, hi[at + j], lo[at + j]);
            } else {
              const float x = __uint_as_float(0x4b000000u | ((w >> (4 * j)) & 15u)) - 8388608.0f;
              const float y = __uint_as_float(0x4b000000u | ((w >> (4 * j + 16)) & 15u)) - 8388608.0f;
              split2(fmaf(x, D, -mn), fmaf(y, D, -mn), hi[at + j], lo[at + j]);
            }
          }
        }
      }
    }
  }
};
template <>
struct Words<QENG_FMT_Q8> {
  uint4 q[2][2];  // [block][quad]
  uint2 s;
  __device__ __forceinline__ void load(uint32_t wbase, uint32_t sbase, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t w0 = wbase + (uint32_t)((g * 4 + (t >> 1)) * 16);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      q[b][0] = lds128(w0 + (uint32_t)(b * 512));
      q[b][1] = lds128(w0 + (uint32_t)(b * 512 + 32));
    }
    s = lds64(sbase + (uint32_t)(g * 8));
  }
  template <int WP>
  __device__ __forceinline__ void dequant(int lane, uint32_t, uint32_t, uint32_t (&hi)[16], uint32_t (&lo)[16]) const {
    // bytes of k = 0,4,1,5 (rows g, g + 8) and of k = 2,6,3,7; a signed byte xor 0x80 under the exponent of 2^23
    const uint32_t s0 = 0x7440u + (lane & 1), s1 = s0 + 2;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const uint32_t s2 = b ? s.y : s.x;
      const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&s2));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 w = q[b][i];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float f = r ? sf.y : sf.x;
          const int at = (b * 2 + i) * 4 + r * 2;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t src = (j ? (r ? w.w : w.z) : (r ? w.y : w.x)) ^ 0x80808080u;
            const float x = __uint_as_float(__byte_perm(src, 0x4b000000u, s0)) - 8388736.0f;
            const float y = __uint_as_float(__byte_perm(src, 0x4b000000u, s1)) - 8388736.0f;
            split2(x * f, y * f, hi[at + j], lo[at + j]);
          }
        }
      }
    }
  }
};

// ---- the same for the epilogues that combine rows r and r + 8 of a 16-row tile (SWIGLU into planes, QKV), of a whole tile -------
// 16 tokens of the warp's 32 rows are turned in shared memory, so that a lane has the 16 rows of one row tile for one token: its
// angles are four loads of 16 bytes, its results one or two stores of 16.  With a lane's row of every token the exchange between
// lanes, the addresses and the 2-byte stores were some 30 instructions a token, which the epilogue's four warps issue between
// those of sixteen dequantising ones: 160 tokens of q|k|v took longer than the tile's MMAs.  1800 tokens (ncu, both in one run):
// q|k|v 6144 x 4096 112 us and 9 for the sums of its cut tiles -> 82 with none cut, gate|up 272 and 7 -> 258; a prompt of 16 x 45
// tokens through 32 layers 9.46 -> 8.07 ms.  (Asking for positions, angles and pages ahead, row by row, gave nothing: 130 us.)
constexpr uint32_t kTurnRow = 36 * 4, kTurnBytes = 4 * 16 * kTurnRow;  // 16 bytes between rows: no bank conflicts either way
__device__ __forceinline__ void drain_pairs(const TcParams& p, int tile, uint32_t rank, uint32_t tacc, int quad, int lane, uint32_t turn) {
  int mt, nt;
  tile_pos(p, tile, mt, nt);
  const int m0 = mt * p.bn, mcnt = min(p.bn, p.M - m0), tl = lane >> 1;
  const int t16 = nt * 16 + (int)rank * 8 + quad * 2 + (lane & 1);  // this lane's row tile, token c0 + tl
  const bool live = t16 * 16 < p.N, swiglu = p.e.kind == QENG_EPI_SWIGLU;
  const qeng_qkv_epi& q = p.e.qkv;
  const int head = t16 >> 3, d = (t16 & 7) << 3, kh = head - q.Hq;
  const bool rotate = !swiglu && head < q.Hq + q.Hkv;
  const uint32_t buf = turn + (uint32_t)quad * (16 * kTurnRow);
  int ps = !swiglu && tl < mcnt && live ? q.pos[m0 + tl] : 0;  // a group ahead
#pragma unroll 1
  for (int c0 = 0; c0 < mcnt; c0 += 16) {
    const int m = c0 + tl;
    bool on = m < mcnt && live;
    float4 cs[4];
    int pid = 0;
    if (!swiglu) {
      if (on && (ps < 0 || ps >= q.max_seq || (ps >> 4) >= q.max_pages)) {
        atomicExch(p.status, 2);
        on = false;
      }
      if (on && rotate) {
        const float4* a = reinterpret_cast<const float4*>(q.cs + (size_t)ps * 128 + d);
        cs[0] = __ldg(a); cs[1] = __ldg(a + 1); cs[2] = __ldg(a + 16); cs[3] = __ldg(a + 17);
      }
      if (on && kh >= 0) pid = q.table[(size_t)((m0 + m) / q.rows_per_seq) * q.max_pages + (ps >> 4)];
    }
    const int at = ps;
    if (!swiglu && m + 16 < mcnt && live) ps = q.pos[m0 + m + 16];
    uint32_t v[16];
    __syncwarp();  // lanes without a token (of the group before) or with a malformed one come from `continue`
    tmem_ld16(tacc + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(buf + (uint32_t)i * kTurnRow + (uint32_t)lane * 4u), "r"(v[i]) : "memory");
    __syncwarp();
    float lo[8], hi[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 w = lds128(buf + (uint32_t)tl * kTurnRow + (uint32_t)((lane & 1) * 64 + i * 16));
      float* const o = i < 2 ? lo + 4 * i : hi + 4 * (i - 2);
      o[0] = __uint_as_float(w.x); o[1] = __uint_as_float(w.y); o[2] = __uint_as_float(w.z); o[3] = __uint_as_float(w.w);
    }
    __syncwarp();
    if (swiglu) {
#pragma unroll
      for (int i = 0; i < 8; ++i) lo[i] = lo[i] / (1.0f + __expf(-lo[i])) * hi[i];
      if (!on) continue;
      __nv_bfloat16* const dst = p.e.yb + (size_t)(m0 + m) * p.e.ldyb + (size_t)t16 * 8;
      uint32_t h[4], l[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) split2(lo[2 * i], lo[2 * i + 1], h[i], l[i]);
      *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
      if (p.e.yb_planes == 2) *reinterpret_cast<uint4*>(dst + p.e.yb_plane) = make_uint4(l[0], l[1], l[2], l[3]);
      continue;
    }
    if (!on) continue;
    if (rotate) {
      const float c[8] = {cs[0].x, cs[0].y, cs[0].z, cs[0].w, cs[1].x, cs[1].y, cs[1].z, cs[1].w};
      const float sn[8] = {cs[2].x, cs[2].y, cs[2].z, cs[2].w, cs[3].x, cs[3].y, cs[3].z, cs[3].w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float a = lo[i], b = hi[i];
        lo[i] = a * c[i] - b * sn[i];
        hi[i] = b * c[i] + a * sn[i];
      }
    }
    __half* dst;
    if (kh < 0) {
      dst = q.q16 + ((size_t)(m0 + m) * q.Hq + head) * 128 + d;
    } else {
      if ((unsigned)pid >= (unsigned)q.pages) {
        atomicExch(p.status, 1);
        continue;
      }
      const int isv = kh >= q.Hkv ? 1 : 0;
      dst = q.pool + (((size_t)pid * q.Hkv + (kh - isv * q.Hkv)) * 2 + isv) * (16 * 128) + (at & 15) * 128 + d;
    }
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 a = __floats2half2_rn(lo[2 * i], lo[2 * i + 1]), b = __floats2half2_rn(hi[2 * i], hi[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&a);
      w[4 + i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(dst + 64) = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// ---- one warp's part of a finished accumulator: groups of 16 tokens from c0 on, every `step` tokens -------------------
// (FIXED: only parts of cut tiles and whole ones added to y)
template <bool FIXED>
__device__ __forceinline__ void drain(const TcParams& p, int tile, bool whole, int pair, uint32_t rank, uint32_t tacc, int quad, int lane, int c0, int step) {
  int mt, nt;
  tile_pos(p, tile, mt, nt);
  const int m0 = mt * p.bn, mcnt = min(p.bn, p.M - m0), row = quad * 32 + lane;
  const int n = nt * 256 + (int)rank * 128 + row;
  qeng_tc_epi e = p.e;
  if (FIXED) e.kind = QENG_EPI_ACCUM;
  auto load = [&](int c, float (&f)[16]) {
    uint32_t v[16];
    tmem_ld16(tacc + ((uint32_t)(quad * 32) << 16) + (uint32_t)c, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
  };
  // Loops without a condition of a lane's own stay whole.  In the last one lanes part where rows lie beyond N (a multiple of 16), or
  // where the epilogue gives them tokens of their own, and are brought together before the next load.  (One loop for all, with
  // that in it: 777 f32 rows over 11008 x 4096 70.1 us, 900 over 22016 x 4096 154.0, 8192 bf16 over 4096 x 11008 590; so 67.7, 145.1,
  // 568.  Rows added to y are no faster in a loop of their own.)
  if (!whole) {
    float* const mine = partial(p, pair, tile - p.dp_tiles, rank, row);
#pragma unroll 1
    for (; c0 < mcnt; c0 += step) {
      float f[16];
      load(c0, f);
#pragma unroll
      for (int i = 0; i < 16; i += 4) __stcg(reinterpret_cast<float4*>(mine + (size_t)(c0 + i) * 128), make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]));
    }
  } else if (!FIXED && e.kind == QENG_EPI_STORE && n - lane + 32 <= p.N) {
#pragma unroll 1
    for (; c0 < mcnt; c0 += step) {
      float f[16];
      load(c0, f);
      float* const dst = e.y + (size_t)(m0 + c0) * e.ldy + n;
      if (mcnt - c0 >= 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[(size_t)i * e.ldy] = f[i];
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i < mcnt - c0) dst[(size_t)i * e.ldy] = f[i];
      }
    }
  } else {
#pragma unroll 1
    for (; c0 < mcnt; c0 += step) {
      float f[16];
      if (e.kind > QENG_EPI_ACCUM || (p.N & 16) != 0) __syncwarp();
      load(c0, f);
      finish<16>(e, p.N, p.status, n, m0 + c0, mcnt - c0, f, lane);
    }
  }
}

// What empties an accumulator: the four epilogue warps row by row; they and the dequantising ones (a single accumulator, added to
// y); or the four by drain_pairs
enum { kPlain = 0, kHelp = 1, kPairs = 2 };
template <int FMT, int WP, int XP, int KST, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                   const __grid_constant__ CUtensorMap smap) {
  constexpr bool HELP = MODE == kHelp;
  constexpr int kW = Fmt<FMT>::kW, kS = Fmt<FMT>::kS;
  constexpr uint32_t kSlot = KST * 8 * (kW + kS), kStageCols = KST * WP * kACols;
  extern __shared__ unsigned char smem_raw[];
  // the swizzle pattern is a function of the address: tiles start on 1024-byte boundaries (the same offset in both CTAs)
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], wfull[kMaxSlots], wempty[kMaxSlots], acc_full[2], acc_empty[2], drained;
  __shared__ uint32_t tmem_slot;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %cluster_ctarank;\n" : "=r"(rank));
  const int pair = blockIdx.x >> 1;
  const uint32_t b_plane = (uint32_t)(p.bn >> 1) * 128u;
  const uint32_t stage_bytes = KST * XP * b_plane;                 // activations: [KST][XP] planes
  const uint32_t ring = smem + (uint32_t)p.nstages * stage_bytes;  // packed-weight slots

  if (tid == 0) {
    for (int s = 0; s < p.nstages; ++s) {
      // the CTA's own set of dequant warps; in the leader also the peer, once its set has arrived there, and the expect_tx
      mbar_init(smem_u32(full + s), kDequantWarps + (rank == 0 ? 2 : 0));
      mbar_init(smem_u32(empty + s), 1);
    }
    for (int s = 0; s < p.nslots; ++s) {
      mbar_init(smem_u32(wfull + s), 1);
      mbar_init(smem_u32(wempty + s), kDequantWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(acc_full + b), 1);
      mbar_init(smem_u32(acc_empty + b), HELP ? 2 * (4 + kHelpers) : 8);  // who empties it, in both CTAs
    }
    mbar_init(smem_u32(&drained), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n");
    // after the allocation: the next kernel may take all of an SM's tensor memory, too, and holds it while it waits for this one
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const uint32_t tmem_a = tmem + (uint32_t)(p.nacc * p.acc_cols);  // the weights' stages, behind the accumulators

  Segments segs(p, pair);
  Seg sg;
  bool failed = false;

  if (warp == 0) {
    if (rank == 0) {
      // ===== MMA issuer =====================================================================
      // f32 accumulate, bf16 x bf16, both K-major, N = bn, M = 256
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | (16u << 24);
      // What the instructions of a stage are issued from has to be warp-uniform for the compiler (votes and shuffles tell it):
      // at 160 columns and less the issue of a stage is as long as its MMAs.
      const uint32_t base = __shfl_sync(0xffffffffu, smem, 0), tm = __shfl_sync(0xffffffffu, tmem, 0), ta = __shfl_sync(0xffffffffu, tmem_a, 0);
      int s = 0, n = 0, buf = 0;
      uint32_t ph = 0, acc_ph = 1;
      while (!failed && segs.next(p, sg)) {
        if (!mbar_wait_cluster(smem_u32(acc_empty + buf), acc_ph)) { failed = true; break; }
        const uint32_t d = tm + (uint32_t)(buf * p.acc_cols);
        uint32_t acc = 0;
        for (int kt = sg.k0; kt < sg.k1; ++kt) {
          if (!mbar_wait_cluster(smem_u32(full + s), ph)) { failed = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          if (elect_one()) {
            const uint32_t a = ta + (uint32_t)s * kStageCols;
            const uint64_t bd = make_desc(base + (uint32_t)s * stage_bytes);
#pragma unroll
            for (int c = 0; c < KST; ++c) {
#pragma unroll
              for (int k = 0; k < kBK / 16; ++k) {  // a K step of 16: 8 columns of A; descriptors count 16-byte units
                const uint32_t ac = a + c * WP * kACols + 8 * k;
                const uint64_t bh = bd + c * XP * (b_plane >> 4) + 2 * k;
                umma_bf16(d, ac, bh, idesc, c > 0 || k > 0 ? 1u : acc);
                if (WP == 2) umma_bf16(d, ac + kACols, bh, idesc, 1u);
                if (XP == 2) umma_bf16(d, ac, bh + (b_plane >> 4), idesc, 1u);
              }
            }
            umma_commit_pair(smem_u32(empty + s));
            if (kt + 1 == sg.k1) umma_commit_pair(smem_u32(acc_full + buf));
          }
          __syncwarp();
          acc = 1;
          if (++s == p.nstages) { s = 0; ph ^= 1u; }
        }
        ++n;
        if (++buf == p.nacc) { buf = 0; acc_ph ^= 1u; }
      }
      // the last accumulators have been read in both CTAs: nothing of this pair is in flight any more
      for (int b = 0; b < p.nacc && b < n; ++b) {
        const int last = n - 1 - b;
        if (!failed && !mbar_wait_cluster(smem_u32(acc_empty + last % p.nacc), (uint32_t)(last / p.nacc) & 1u)) failed = true;
      }
      if (failed) {  // what was issued still has to finish before tensor memory is freed
        if (elect_one()) umma_commit_pair(smem_u32(&drained));
        __syncwarp();
        mbar_wait(smem_u32(&drained), 0);
        if (lane == 0) atomicExch(p.status, 4);
      }
    } else {
      // ===== the peer's weights: one arrival at the leader per stage, for the eight of its warps =========
      const int total = segs.stages(p);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < total; ++i) {
        if (!mbar_wait(smem_u32(full + s), ph)) failed = true;
        if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\ntcgen05.fence::before_thread_sync;\n" ::: "memory");
        if (lane == 0) mbar_arrive_cluster(map_leader(smem_u32(full + s)));
        if (++s == p.nstages) { s = 0; ph ^= 1u; }
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
          if (rank == 0) mbar_expect_tx(smem_u32(full + s), 2 * stage_bytes);
          const uint32_t b = smem + (uint32_t)s * stage_bytes, bar = map_leader(smem_u32(full + s));
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
    // (whose tensor-memory lanes lie in the quadrant that this warp may write, warp % 4)
    const int set = (warp - 8) >> 3, rt = (warp & 3) * 2 + ((warp >> 2) & 1);
    const uint32_t dst0 = tmem_a + ((uint32_t)(rt * 16) << 16);
    const uint32_t wb0 = ring + (uint32_t)rt * (KST * kW), sb0 = ring + 8u * KST * kW + (uint32_t)rt * (KST * kS);
    const uint32_t mask = in_register(0x000f000fu), base = in_register(0x43004300u);
    const int total = segs.stages(p);
    // Whoever waits on a barrier by parity has to see all of its phases (boxes may land out of order: a set that skipped
    // one could take the phase before the last for the one it needs), so the number of packed slots is even and a slot
    // always belongs to one set.  (Stages need no such care: two stages ago this set waited for a consumption no
    // earlier than the one before the last of this stage, and the MMAs consume in order.)
    int s = set, ws = set;
    uint32_t ph = 1, wph = 0;
    // HELP: one accumulator, added to y.  The MMAs stand still while it is emptied, and so would these warps as soon as all
    // stages are full: they take four fifths of it instead, as it is the latency of the old values that makes it long.  A segment
    // is due once the stage ahead (i) is one that the first stage of the next segment has to free; up to there a warp has filled
    // all that the segment's MMAs need.  4096 rows bf16 over 22016 x 4096 803 -> 633 us, over 4096 x 4096 152 -> 123, 1800 rows
    // over 4096 x 11008 149 -> 134.  (Stores and parts are no faster for it: those are bound by the way to L2.)
    bool owed = HELP && segs.next(p, sg);
    int due = owed ? sg.k1 - sg.k0 + p.nstages : 0;
    uint32_t acc_ph = 0;
    for (int i = set;;) {
      const int stop = owed ? min(total, due) : total;
#pragma unroll 1
      for (; i < stop; i += kSets) {
        if (!failed && !mbar_wait(smem_u32(wfull + ws), wph)) failed = true;
        const uint32_t wb = wb0 + (uint32_t)ws * kSlot, sb = sb0 + (uint32_t)ws * kSlot, at = dst0 + (uint32_t)s * kStageCols;
        Words<FMT> w[KST];
#pragma unroll
        for (int c = 0; c < KST; ++c) w[c].load(wb + (uint32_t)(c * kW), sb + (uint32_t)(c * kS), lane);
#pragma unroll
        for (int c = 0; c < KST; ++c) {
          uint32_t hi[16], lo[16];
          w[c].template dequant<WP>(lane, mask, base, hi, lo);
          if (c == 0) {
            if (!failed && !mbar_wait(smem_u32(empty + s), ph)) failed = true;
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          }
          tmem_st16(at + (uint32_t)(c * WP * kACols), hi);
          if (WP == 2) tmem_st16(at + (uint32_t)(c * WP * kACols + kACols), lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\ntcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(smem_u32(full + s));
          mbar_arrive(smem_u32(wempty + ws));
        }
        if ((s += kSets) >= p.nstages) { s -= p.nstages; ph ^= 1u; }
        if ((ws += kSets) >= p.nslots) { ws -= p.nslots; wph ^= 1u; }
      }
      if (!owed) break;
      asm volatile("griddepcontrol.wait;\n" ::: "memory");
      if (!failed && !mbar_wait(smem_u32(acc_full), acc_ph)) failed = true;
      acc_ph ^= 1u;
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const bool whole = sg.k0 == 0 && sg.k1 == p.nk;
      if (!__any_sync(0xffffffffu, failed) && whole)
        drain<true>(p, sg.tile, whole, pair, rank, tmem, warp & 3, lane, 16 * (1 + ((warp - 8) >> 2)), 16 * (1 + kHelpers / 4));
      __syncwarp();
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_leader(smem_u32(acc_empty)));
      owed = segs.next(p, sg);
      if (owed) due += sg.k1 - sg.k0;
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
  } else if (warp >= 4) {
    // ===== epilogue: warp = one quadrant of tensor-memory lanes =====================================
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int quad = warp & 3;
    int buf = 0;
    uint32_t acc_ph = 0;
    while (segs.next(p, sg)) {
      const bool whole = sg.k0 == 0 && sg.k1 == p.nk;
      if (!failed && !mbar_wait(smem_u32(acc_full + buf), acc_ph)) failed = true;
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      if (!__any_sync(0xffffffffu, failed)) {
        if (MODE == kPairs && whole) drain_pairs(p, sg.tile, rank, tmem + (uint32_t)(buf * p.acc_cols), quad, lane, ring + (uint32_t)p.nslots * kSlot);
        else drain<HELP || MODE == kPairs>(p, sg.tile, whole, pair, rank, tmem + (uint32_t)(buf * p.acc_cols), quad, lane, 0, HELP && whole ? 16 * (1 + kHelpers / 4) : 16);
      }
      __syncwarp();
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_leader(smem_u32(acc_empty + buf)));
      if (++buf == p.nacc) { buf = 0; acc_ph ^= 1u; }
    }
    if (failed && lane == 0) atomicExch(p.status, 4);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  if (__syncthreads_or(failed)) grace();
  cluster_sync();  // no CTA leaves while its peer may still signal it or read its shared memory
  if (warp == 3) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
}

// ---- tiles cut along K: the parts, added in K order, through the epilogue -----------------------------------
// Grid: (split tile, CTA of the pair) x kSumTokens tokens; thread = weight row.  Its time is the latency of the parts (2 to 6 of
// a tile): three are requested together.  f32 rows, one part at a time / so: 101 over 4096 x 4096 23.9 / 20.9 us a call, 240 over
// 11008 x 4096 57.1 / 56.9; 8 tokens a thread 20.4 / 58.0, 4 tokens 20.0 / 61.3 (a CTA's start costs more than its sums).
constexpr int kSumTokens = 16, kSumAhead = 3;
__global__ void __launch_bounds__(128) tc_reduce_kernel(const TcParams p) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int r = blockIdx.x >> 1, rank = blockIdx.x & 1, c0 = blockIdx.y * kSumTokens, row = threadIdx.x;
  const long long U = (long long)p.sk_tiles * p.nk;
  int mt, nt;
  tile_pos(p, p.dp_tiles + r, mt, nt);
  const int m0 = mt * p.bn, mcnt = min(p.bn, p.M - m0);
  const int q0 = pair_of_unit(U, p.npairs, r * p.nk), q1 = pair_of_unit(U, p.npairs, (r + 1) * p.nk - 1);
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  if (q0 == q1 || c0 >= mcnt) return;  // one pair had all of K: its epilogue is done
  float f[kSumTokens];
#pragma unroll
  for (int i = 0; i < kSumTokens; ++i) f[i] = 0.f;
  for (int q = q0; q <= q1; q += kSumAhead) {
    float4 v[kSumAhead][kSumTokens / 4];
#pragma unroll
    for (int j = 0; j < kSumAhead; ++j) {
      const float4* src = reinterpret_cast<const float4*>(partial(p, min(q + j, q1), r, (uint32_t)rank, row) + (size_t)c0 * 128);
#pragma unroll
      for (int i = 0; i < kSumTokens / 4; ++i) v[j][i] = __ldcg(src + i * 128);
    }
#pragma unroll
    for (int j = 0; j < kSumAhead; ++j) {
      if (q + j > q1) break;
#pragma unroll
      for (int i = 0; i < kSumTokens / 4; ++i) {
        f[4 * i] += v[j][i].x;
        f[4 * i + 1] += v[j][i].y;
        f[4 * i + 2] += v[j][i].z;
        f[4 * i + 3] += v[j][i].w;
      }
    }
  }
  finish<kSumTokens>(p.e, p.N, p.status, nt * 256 + rank * 128 + row, m0 + c0, mcnt - c0, f, row & 31);
}

// ---- activation rows -> one or two bf16 planes, optionally RMS-normalised on the way ----------------------
// One CTA per row, or several (grid.y) where no norm has to see the whole row: with a few rows the chain of loads of
// one CTA is the time (16 rows x 11008: 6 us with a row to a CTA, 2 us split).  With many rows the time is the chain of a row (loads,
// the sum of its squares, stores) times the rounds of CTAs on an SM: 256 threads with four loads of 16 bytes on their way each take
// 4096 values at once and leave room for 5 or 6 rows on an SM at 48 or 40 registers, where 512 threads had half of their registers
// idle and room for 4 (ncu: a norm of 1800 rows 15.4 -> 13.3 us; the call of a prompt of 1800 tokens 21.20 -> 21.08 ms; the
// conversion of 777 f32 rows is no faster for it).  Up to two rows to an SM, 512 threads are the shorter chain (45-token prompts and
// 24 tokens of 16 sequences: 71.6 ms, with 256 threads 72.7).
constexpr int kPrepMany = 256, kPrepFew = 512;
constexpr int kPrepKeep = 4;  // loads of a thread in flight
template <bool NORM, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kPrepFew ? 2 : NORM ? 5 : 6) tc_prep_kernel(const void* __restrict__ x, int dtype, long long ldx, int K,
                                                      const float* __restrict__ gamma, float eps,
                                                      __nv_bfloat16* __restrict__ out, long long plane, int planes,
                                                      float* __restrict__ sums, int sum_blocks) {
  __shared__ float sh[THREADS / 32];
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (NORM)  // the weights of a layer pass through L2 between two uses of its gains
    for (int k = threadIdx.x * 8; k < K; k += 8 * THREADS) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(gamma + k));
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int tid = threadIdx.x;
  const long long row = blockIdx.x;
  // K is a multiple of 32; a row of f32 may start at any 4-byte boundary
  const bool vec = dtype == QENG_F32 && ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ldx * 4)) & 15) == 0;
  const bool gvec = NORM && (reinterpret_cast<uintptr_t>(gamma) & 15) == 0;
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
  auto emit = [&](int k, float (&v)[4]) {  // whole warps: the block sums are shuffled
    uint2 hi = make_uint2(0u, 0u), lo = make_uint2(0u, 0u);
    if (k < K) {
      if (NORM) {
        float g[4];
        if (gvec) {
          const float4 a = *reinterpret_cast<const float4*>(gamma + k);
          g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) g[i] = gamma[k + i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = v[i] * rs * g[i];
      }
      split2(v[0], v[1], hi.x, lo.x);
      split2(v[2], v[3], hi.y, lo.y);
      *reinterpret_cast<uint2*>(out + row * K + k) = hi;
      if (planes == 2) *reinterpret_cast<uint2*>(out + plane + row * K + k) = lo;
    }
    if (sums != nullptr) {  // per 32-block and plane, the sum of the values as stored (K-quant blocks: the minimum's factor)
      auto sum4 = [](uint2 u) {
        const float2 a = __bfloat1622float2(bf2(u.x)), b = __bfloat1622float2(bf2(u.y));
        float t = (a.x + a.y) + (b.x + b.y);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 4);
        return t;
      };
      const float sh0 = sum4(hi), sl0 = sum4(lo);
      const int blk = k >> 5;
      if ((tid & 7) == 0 && blk < sum_blocks) {
        sums[row * sum_blocks + blk] = sh0;
        if (planes == 2) sums[((long long)gridDim.x + row) * sum_blocks + blk] = sl0;
      }
    }
  };
  constexpr int kKeep = NORM || THREADS == kPrepMany ? kPrepKeep : 1;  // few rows: a thread has one load, see `parts`
  float v[kKeep][4];
  if (!NORM) {
    const int step = 4 * THREADS * (int)gridDim.y;
    for (int k0 = ((int)blockIdx.y * THREADS + tid) * 4; (k0 & ~127) < K; k0 += kKeep * step) {
#pragma unroll
      for (int j = 0; j < kKeep; ++j) {
        const int k = k0 + j * step;
        v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
        if (k < K) load4(k, v[j]);
      }
#pragma unroll
      for (int j = 0; j < kKeep; ++j) {
        const int k = k0 + j * step;
        if ((k & ~127) < K) emit(k, v[j]);
      }
    }
    return;
  }
  // the first kKeep * 4 * THREADS values of the row stay in registers across the reduction
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kKeep; ++j) {
    const int k = (j * THREADS + tid) * 4;
    v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
    if (k < K) load4(k, v[j]);
  }
#pragma unroll
  for (int j = 0; j < kKeep; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = fmaf(v[j][i], v[j][i], ss);
  for (int k = (kKeep * THREADS + tid) * 4; k < K; k += 4 * THREADS) {
    float w[4];
    load4(k, w);
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = fmaf(w[i], w[i], ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) sh[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w) tot += sh[w];
  rs = rsqrtf(tot / (float)K + eps);
#pragma unroll
  for (int j = 0; j < kKeep; ++j) {
    const int k = (j * THREADS + tid) * 4;
    if ((k & ~127) < K) emit(k, v[j]);
  }
  for (int k = (kKeep * THREADS + tid) * 4; (k & ~127) < K; k += 4 * THREADS) {
    float w[4] = {};
    if (k < K) load4(k, w);
    emit(k, w);
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

// As many stages as tensor memory holds of the weights and shared memory of the activations, beside four slots of packed
// weights; what is left goes to the packed ring (few tokens: the weights come from HBM and want tens of KB in flight, and then a
// stage leaves room for it).  False where two stages do not fit.
bool fit_rings(Plan* pl, int fmt, int wp, int xp) {
  const size_t stage = (size_t)pl->kst * xp * (pl->bn / 2) * 128, slot = (size_t)slot_bytes_of(fmt, pl->kst);
  const size_t turn = pl->pairs ? kTurnBytes : 0, room = kSmemBudget - 1024 - 1024 - turn;  // alignment, static shared memory
  pl->nstages = std::min(std::min((512 - pl->nacc * pl->acc_cols) / (pl->kst * wp * kACols), kMaxStages), (int)((room - 4 * slot) / stage));
  if (pl->nstages < 2) return false;
  pl->nslots = (int)((room - pl->nstages * stage) / slot);
  pl->nslots = (pl->nslots < kMaxSlots ? pl->nslots : kMaxSlots) / kSets * kSets;  // a slot belongs to one dequant set
  pl->smem = pl->nstages * stage + pl->nslots * slot + turn + 1024;
  return true;
}

// Tile width, stages and split, by a cost model in cycles.  Its constants were fitted to 1265 calls (three formats, f32 and bf16
// rows, 17 to 4096 of them, seven matrices, store and accumulate) and to 68 prompts, each timed with every plan that fits: the
// plan it picks takes 1.0 % longer than the best one in the mean.  Per 64 k:
//   the MMAs take 2 * bn per product, the dequantisation 430 (4-bit blocks, one term), 735 (two), 870 (8-bit) or 1020 (K-quant),
//   a stage what is longer; stages of one chunk add 34 to the former and 76 to the latter (each has its barriers), two stages in
//   all 106 and 163 (one waits for the other's refill).
// Emptying an accumulator takes 17 cycles a token (store), 27 (accumulate), 12 with the dequantising warps' help, 100 (SWIGLU row by
// row) and 250 (QKV row by row), 60 of both by drain_pairs (fitted to K of 4096: 40, 60, 80, 90 and 100 for either, prompts of 45 to
// 1800 tokens); the next tile hides it where there are two of them (a last store then takes 11).  Two terms over K below 2048 count
// the former two although drain_pairs empties their whole tiles as well: with 60 the plans of layers 1024 to 1920 wide come out up to
// 6 % slower (101 and 128 tokens, 4000 of 8-bit blocks: cut tiles are then worth more than the model has them), those of 256 and 512
// up to 15 % faster.  One term takes 60 at every K: 300 to 4000 tokens through layers 256 to 1920 wide take 2 to 23 % less than with
// 100 and 250 (1024 wide, 1400 tokens 175 -> 147 us a layer; 1920 wide, 1000 tokens 195 -> 191), none more.
// Every tile of the first round costs 29 (the pairs' first loads meet).  Tiles cut along K pay for their parts (64 a token,
// 0.6 of it where another segment hides one), their sums (700 a part) and the second launch (9400).
Plan make_plan(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int wp, int xp, int epi, bool pairs_ok, bool may_split) {
  Plan best = {};
  double best_cost = 1e30;
  const int pairs = ctx->sm_count / 2, n_tiles = (int)((w->N + 255) / 256), products = wp + xp - 1;
  const double deq = w->fmt == QENG_FMT_Q4 ? (wp == 1 ? 430 : 735) : w->fmt == QENG_FMT_Q8 ? 870 : 1020;
  const int widest = M <= 256 ? (int)((M + 15) / 16 * 16) : 256, narrowest = M <= 128 ? widest : 80;
  for (int bn = widest; bn >= narrowest; bn -= 16) {
    for (int form = 0; form < (wp == 1 ? 2 : 4); ++form) {  // stages of two chunks or (two terms) of one; one accumulator or two
      Plan c = {};
      c.kst = form < 2 ? 2 : 1;
      c.nacc = 1 + form % 2;
      c.acc_cols = (bn + 31) / 32 * 32;
      c.bn = bn;
      c.pairs = pairs_ok;
      if (!fit_rings(&c, w->fmt, wp, xp)) continue;
      c.m_tiles = (int)((M + bn - 1) / bn);
      c.n_tiles = n_tiles;
      c.nk = (int)((w->nchunks + c.kst - 1) / c.kst);
      const int T = c.m_tiles * n_tiles, waves = (T + pairs - 1) / pairs, rem = T % pairs, nk = c.nk;
      const bool two = c.nstages == 2, one = c.kst == 1;
      const double mma = 2.0 * c.kst * std::max(bn, 32) * products + (one ? 34 : 0) + (two ? 106 : 0);
      const double convert = c.kst * deq + (one ? 76 : 0) + (two ? 163 : 0);
      const double stage = std::max(mma, convert);
      const bool turned = pairs_ok && (wp == 1 || w->nchunks >= 32);
      const double per_token = epi == QENG_EPI_QKV ? (turned ? 60 : 250) : epi == QENG_EPI_SWIGLU ? (turned ? 60 : 100) : epi == QENG_EPI_STORE ? (c.nacc == 1 ? 17 : 11) : c.nacc == 1 ? 12 : 27;
      const double ep = per_token * bn, body = nk * stage, tile = c.nacc == 1 ? body + ep : std::max(body, ep);
      const double dp = waves * tile + (c.nacc == 1 ? 0.0 : ep) + 29.0 * std::min(T, pairs);
      // shares of at least two stages (with no whole tiles the number of pairs is reduced instead)
      const int sharing = T < pairs ? std::min(pairs, std::max(1, (int)((int64_t)rem * nk / 2))) : pairs;
      const double share = (double)rem * nk / sharing, parts = 1 + std::max(1.0, nk / std::max(share, 1.0));
      // the share of a cut tile has to hide the epilogue of the pair's last whole one, old values of y from HBM among it
      const double tail = c.nacc == 1 || T < pairs ? 0.0 : std::max(0.0, (epi == QENG_EPI_ACCUM ? 100 : per_token) * bn - share * stage);
      // (whole and cut tiles added to y took 1.5 to 5 us more than stored ones, cut tiles alone 1)
      const double mixed = epi == QENG_EPI_ACCUM && T >= pairs ? 4000.0 : 0.0;
      const double sk = (T / pairs) * tile + share * stage + tail + mixed + (c.nacc == 1 ? 64.0 : 38.0) * bn + 700 * parts + 9400;
      const bool cut = may_split && rem != 0 && sk < dp && (T < pairs || (int64_t)rem * nk >= 2 * (int64_t)pairs);
      const double cost = cut ? sk : dp;
      if (cost >= best_cost) continue;
      best_cost = cost;
      c.sk_tiles = cut ? rem : 0;
      c.dp_tiles = T - c.sk_tiles;
      c.npairs = cut ? sharing : std::min(T, pairs);
      best = c;
    }
  }
  if (best.pairs && best.dp_tiles == 0) {  // (nothing but parts, whose sums another kernel finishes: their room goes to the packed ring)
    best.pairs = false;
    fit_rings(&best, w->fmt, wp, xp);
  }
  best.box_rows = best.bn / 2;
  best.ws_floats = best.sk_tiles > 0 ? (size_t)best.npairs * 4 * best.bn * 128 : 0;
  return best;
}

// tensor maps of the packed planes, boxes of kst chunks x 8 row tiles of 64-bit words; kept with the weight
bool weight_maps(const qeng_weight* w) {
  std::lock_guard<std::mutex> hold(w->lock);
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

template <int FMT, int WP, int XP, int KST, int MODE>
int32_t launch(qeng_ctx* ctx, const qeng_weight* w, const TcParams& p, const Plan& pl, const CUtensorMap& map, cudaStream_t stream) {
  static bool configured_on[64] = {};  // the opt-in shared-memory size is set per device
  bool& configured = configured_on[ctx->device & 63];
  if (!configured) {
    QENG_CUDA(ctx, cudaFuncSetAttribute(gemm_tc_kernel<FMT, WP, XP, KST, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
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
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, gemm_tc_kernel<FMT, WP, XP, KST, MODE>, p, map, *wm, *sm));
  return p.sk_tiles > 0 ? reduce(ctx, p, stream) : QENG_OK;
}

}  // namespace

int32_t qeng_tc::prepare(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, const qeng_tc_epi& epi, qeng_scratch* sc,
                         const Plan* pl, TcParams* p, CUtensorMap* map) {
  if ((reinterpret_cast<uintptr_t>(x.data) & 15) != 0 || (x.ld & 7) != 0)
    return qeng_fail(ctx, QENG_ERR_ALIGN, "gemm_tc: activations must be 16-byte aligned with a leading dimension multiple of 8");
  p->ws = nullptr;
  if (pl->sk_tiles > 0) {
    const int32_t rc = qeng_scratch_grow(ctx, sc, &sc->part, pl->ws_floats * 4);
    if (rc != QENG_OK) return ctx->no_memory ? QENG_ERR_STATE : rc;
    p->ws = reinterpret_cast<float*>(sc->part.ptr);
  }
  EncodeFn enc = encode_fn();
  if (!enc || !weight_maps(w)) return qeng_fail(ctx, QENG_ERR_CUDA, "gemm_tc: cuTensorMapEncodeTiled is not available or rejects the packed planes");
  const cuuint64_t dims[3] = {(cuuint64_t)w->K, (cuuint64_t)M, (cuuint64_t)x.planes};
  const cuuint64_t strides[2] = {(cuuint64_t)x.ld * 2, (cuuint64_t)(x.planes > 1 ? x.plane : x.ld * M) * 2};
  const cuuint32_t box[3] = {kBK, (cuuint32_t)pl->box_rows, 1}, es[3] = {1, 1, 1};
  if (enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(x.data), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return qeng_fail(ctx, QENG_ERR_CUDA, "gemm_tc: tensor map rejected (M=%lld, K=%lld, ld=%lld)", (long long)M, (long long)w->K, (long long)x.ld);
  p->nk = pl->nk; p->M = (int)M; p->N = (int)w->N;
  p->bn = pl->bn; p->m_tiles = pl->m_tiles; p->n_tiles = pl->n_tiles; p->dp_tiles = pl->dp_tiles; p->sk_tiles = pl->sk_tiles;
  p->nstages = pl->nstages; p->nslots = pl->nslots; p->nacc = pl->nacc; p->acc_cols = pl->acc_cols; p->npairs = pl->npairs; p->e = epi;
  p->status = ctx->status;
  return QENG_OK;
}

int32_t qeng_tc::reduce(qeng_ctx* ctx, const TcParams& p, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * p.sk_tiles), (unsigned)(p.bn / kSumTokens));
  cfg.blockDim = dim3(128);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, tc_reduce_kernel, p));
  return QENG_OK;
}

void* qeng_tensor_map_encoder() { return reinterpret_cast<void*>(encode_fn()); }

int32_t qeng_tc_prep(qeng_ctx* ctx, const void* x, int32_t dtype, int64_t M, int64_t K, int64_t ldx, const float* gamma, float eps,
                     int planes, void* out, float* sums, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  const bool few = M < 2 * ctx->sm_count;
  const int threads = few ? kPrepFew : kPrepMany;
  const int64_t parts = gamma == nullptr && few ? (K + 4 * threads - 1) / (4 * threads) : 1;
  cfg.gridDim = dim3((unsigned)M, (unsigned)parts);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  auto* kernel = gamma != nullptr ? (few ? tc_prep_kernel<true, kPrepFew> : tc_prep_kernel<true, kPrepMany>)
                                  : (few ? tc_prep_kernel<false, kPrepFew> : tc_prep_kernel<false, kPrepMany>);
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, x, (int)dtype, (long long)ldx, (int)K, gamma, eps,
                                    reinterpret_cast<__nv_bfloat16*>(out), (long long)(M * K), planes, sums,
                                    (int)((K / 32 + 1) / 2 * 2)));
  return QENG_OK;
}

int32_t qeng_gemm_tc(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, int wp, const qeng_tc_epi& epi, cudaStream_t stream, qeng_scratch* sc) {
  const int xp = x.planes;
  if (w->fmt != QENG_FMT_Q4 && wp == 1) return qeng_fail(ctx, QENG_ERR_SHAPE, "gemm_tc: single bf16 weights are for 4-bit blocks only");
  if (wp == 1 && xp != 1) return qeng_fail(ctx, QENG_ERR_ARG, "gemm_tc: two activation planes need two weight planes");
  // drain_pairs makes 16-byte accesses: rows of planes, pages and angles allow them (the decoder's buffers)
  const bool pairs_ok = epi.kind == QENG_EPI_QKV || (epi.kind == QENG_EPI_SWIGLU && epi.yb != nullptr &&
                        ((reinterpret_cast<uintptr_t>(epi.yb) | (uintptr_t)(epi.ldyb * 2) | (uintptr_t)(epi.yb_plane * 2)) & 15) == 0);
  Plan pl = make_plan(ctx, w, M, wp, xp, epi.kind, pairs_ok, true);
  TcParams p;
  CUtensorMap map;
  if (pl.sk_tiles > 0 && sc == nullptr) sc = qeng_scratch_for(ctx, stream);
  int32_t rc = prepare(ctx, w, x, M, epi, sc, &pl, &p, &map);
  if (rc == QENG_ERR_STATE) {  // no memory for the workspace: whole tiles only
    pl = make_plan(ctx, w, M, wp, xp, epi.kind, pairs_ok, false);
    rc = prepare(ctx, w, x, M, epi, sc, &pl, &p, &map);
  }
  if (rc != QENG_OK) return rc;
  const bool help = pl.nacc == 1 && epi.kind == QENG_EPI_ACCUM;
#define QENG_TC_M(F, W, X, K)                                                 \
  (help ? launch<F, W, X, K, kHelp>(ctx, w, p, pl, map, stream)               \
        : pl.pairs ? launch<F, W, X, K, kPairs>(ctx, w, p, pl, map, stream) : launch<F, W, X, K, kPlain>(ctx, w, p, pl, map, stream))
  if (wp == 1) return QENG_TC_M(QENG_FMT_Q4, 1, 1, 2);
#define QENG_TC_K(F, X, K) QENG_TC_M(F, 2, X, K)
#define QENG_TC(F, X) (pl.kst == 2 ? QENG_TC_K(F, X, 2) : QENG_TC_K(F, X, 1))
  switch (w->fmt) {
    case QENG_FMT_Q4: return xp == 1 ? QENG_TC(QENG_FMT_Q4, 1) : QENG_TC(QENG_FMT_Q4, 2);
    case QENG_FMT_Q8: return xp == 1 ? QENG_TC(QENG_FMT_Q8, 1) : QENG_TC(QENG_FMT_Q8, 2);
    default: return xp == 1 ? QENG_TC(QENG_FMT_K4, 1) : QENG_TC(QENG_FMT_K4, 2);
  }
#undef QENG_TC
#undef QENG_TC_K
#undef QENG_TC_M
}

// y[M,N] = x . dequant(W)^T through the kernel above, activations in any type the entry point takes.
// wp = 1: operands rounded to bf16; wp = 2: two bf16 terms per weight and per f32 / f16 activation.
int32_t qeng_gemm_many_rows(qeng_ctx* ctx, const qeng_weight* w, const void* x, int32_t x_dtype, int64_t M, int64_t ldx, qeng_tc_epi e, int wp,
                            cudaStream_t stream) {
  float* const y = e.y;
  const int planes = wp == 1 || x_dtype == QENG_BF16 ? 1 : 2;
  qeng_tc_x xx;
  if (x_dtype == QENG_BF16 && ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ldx * 2)) & 15) == 0) {
    xx.data = x;
    xx.ld = ldx;
    return qeng_gemm_tc(ctx, w, xx, M, wp, e, stream);
  }
  // the planes of one pass take a gigabyte at most (or those of 256 rows, if that is more)
  const int64_t row_bytes = (int64_t)planes * w->K * 2, most = std::max<int64_t>(256, ((int64_t)1 << 30) / row_bytes);
  const int64_t passes = (M + most - 1) / most, step = (M + passes - 1) / passes;
  qeng_scratch* sc = qeng_scratch_for(ctx, stream);
  int32_t rc = qeng_scratch_grow(ctx, sc, &sc->planes, (size_t)(step * row_bytes));
  for (int64_t m0 = 0; rc == QENG_OK && m0 < M; m0 += step) {
    const int64_t rows = std::min(step, M - m0);
    const char* src = reinterpret_cast<const char*>(x) + m0 * ldx * (x_dtype == QENG_F32 ? 4 : 2);
    rc = qeng_tc_prep(ctx, src, x_dtype, rows, w->K, ldx, nullptr, 0.f, planes, sc->planes.ptr, nullptr, stream);
    xx.data = sc->planes.ptr; xx.planes = planes; xx.ld = w->K; xx.plane = rows * w->K;
    e.y = y + m0 * e.ldy;
    if (rc == QENG_OK) rc = qeng_gemm_tc(ctx, w, xx, rows, wp, e, stream, sc);
  }
  return rc;
}

// For the tests, which have to meet every kind of plan: chunks a stage, tokens a tile, accumulators, whole tiles, cut tiles, pairs.
extern "C" int32_t qeng_many_rows_plan(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int32_t wp, int32_t xp, int32_t epilogue, int32_t* out) {
  const Plan pl = make_plan(ctx, w, M, wp, xp, epilogue, epilogue == QENG_EPI_QKV || epilogue == QENG_EPI_SWIGLU, true);
  const int v[6] = {pl.kst, pl.bn, pl.nacc, pl.dp_tiles, pl.sk_tiles, pl.npairs};
  std::copy(v, v + 6, out);
  return QENG_OK;
}
