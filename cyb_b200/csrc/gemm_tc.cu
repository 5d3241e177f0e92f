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
#include <algorithm>

#include "gemm_tc.cuh"

namespace {
using namespace qeng_tc;

constexpr int kDequantWarps = 8;         // per set
constexpr int kThreads = (8 + 2 * kDequantWarps) * 32;

// ---- dequantisation: one lane's words of one 32-block -> rows g and g+8, 8 consecutive k each ------------------
// The inner loop of the kernel: its rate is set by the integer pipe (half rate), so the 4-bit form spends two
// integer instructions per pair of weights (shift, AND-OR) and leaves the rest to the FMA pipe.
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

template <int FMT, int WP, int XP, int KST>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                   const __grid_constant__ CUtensorMap smap) {
  constexpr int kW = Fmt<FMT>::kW, kS = Fmt<FMT>::kS;
  constexpr uint32_t kSlot = KST * 8 * (kW + kS);
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
    mbar_init(smem_u32(&drained), 1);
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
      while (!failed && segs.next(p, sg)) {
        const int buf = n & 1;
        for (int kt = sg.k0; kt < sg.k1; ++kt) {
          if (kt == sg.k0 && !mbar_wait(smem_u32(acc_empty + buf), (((uint32_t)n >> 1) & 1u) ^ 1u)) failed = true;
          if (failed || !mbar_wait(smem_u32(full + s), ph)) failed = true;
          if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          // (the shuffles tell the compiler what is warp-uniform: MMA operands live in uniform registers)
          const uint32_t a = __shfl_sync(0xffffffffu, smem + (uint32_t)s * stage_bytes, 0);
          const uint32_t d = __shfl_sync(0xffffffffu, tmem + (uint32_t)buf * 256u, 0);
          if (elect_one()) {
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
      if (failed) {  // what was issued still has to finish before tensor memory is freed
        if (elect_one()) umma_commit_pair(smem_u32(&drained));
        __syncwarp();
        mbar_wait(smem_u32(&drained), 0);
        if (lane == 0) atomicExch(p.status, 4);
      }
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
        // Whoever waits on a barrier by parity has to see all of its phases (boxes may land out of order: a set that
        // skipped one could take the phase before the last for the one it needs), so the number of packed slots is
        // even and a slot always belongs to one set.  (Operand stages need no such care: two stages ago this set waited
        // for a consumption later than the one before the last of this stage, and the MMAs consume in order.)
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
          finish<16>(p.e, p.N, p.status, wrow, m0 + c0, mcnt - c0, f, lane);
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
  if (__syncthreads_or(failed)) grace();
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
  finish<16>(p.e, p.N, p.status, nt * 256 + rank * 128 + row, m0 + c0, mcnt - c0, f, row & 31);
}

// ---- activation rows -> one or two bf16 planes, optionally RMS-normalised on the way ----------------------
// One CTA per row, or several (grid.y) where no norm has to see the whole row: with a few rows the chain of loads of
// one CTA is the time (16 rows x 11008: 6 us with 256 threads a row, 2 us split).
constexpr int kPrepThreads = 512;
__global__ void __launch_bounds__(kPrepThreads) tc_prep_kernel(const void* __restrict__ x, int dtype, long long ldx, int K,
                                                      const float* __restrict__ gamma, float eps,
                                                      __nv_bfloat16* __restrict__ out, long long plane, int planes,
                                                      float* __restrict__ sums, int sum_blocks) {
  __shared__ float sh[kPrepThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (gamma != nullptr)  // the weights of a layer pass through L2 between two uses of its gains
    for (int k = threadIdx.x * 8; k < K; k += 8 * kPrepThreads) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(gamma + k));
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
  auto emit = [&](int k, float (&v)[4]) {  // whole warps: the block sums are shuffled
    uint2 hi = make_uint2(0u, 0u), lo = make_uint2(0u, 0u);
    if (k < K) {
      if (gamma != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = v[i] * rs * gamma[k + i];
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
  if (gamma == nullptr) {
    for (int k = ((int)blockIdx.y * kPrepThreads + tid) * 4; (k & ~127) < K; k += 4 * kPrepThreads * (int)gridDim.y) {
      float v[4] = {};
      if (k < K) load4(k, v);
      emit(k, v);
    }
    return;
  }
  // the first kKeep * 2048 values of the row stay in registers across the reduction
  constexpr int kKeep = 4;
  float v[kKeep][4], ss = 0.f;
#pragma unroll
  for (int j = 0; j < kKeep; ++j) {
    const int k = (j * kPrepThreads + tid) * 4;
    v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
    if (k < K) load4(k, v[j]);
  }
#pragma unroll
  for (int j = 0; j < kKeep; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = fmaf(v[j][i], v[j][i], ss);
  for (int k = (kKeep * kPrepThreads + tid) * 4; k < K; k += 4 * kPrepThreads) {
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
  for (int w = 0; w < kPrepThreads / 32; ++w) tot += sh[w];
  rs = rsqrtf(tot / (float)K + eps);
#pragma unroll
  for (int j = 0; j < kKeep; ++j) {
    const int k = (j * kPrepThreads + tid) * 4;
    if ((k & ~127) < K) emit(k, v[j]);
  }
  for (int k = (kKeep * kPrepThreads + tid) * 4; (k & ~127) < K; k += 4 * kPrepThreads) {
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

// Up to this many tokens two stages of two chunks, both operands in two terms, fit shared memory beside the packed ring of
// every block format.  (8-bit blocks set it: 4-bit and K-quant blocks would fit up to 144 tokens, bf16 rows, which have one
// term, up to 240 and more.)
constexpr int64_t kWideStage = 112;

// Tile width and split, by a cost model in cycles.  Per 64 k the MMAs take 2 * bn per product and the dequantisation a
// fixed time, whichever is longer; tiles cut along K pay for their partials' way through L2 and a second launch.  The fixed
// times are what its instructions take to issue.  The stages are slower than that, since the steps of a stage depend on
// one another: 1320 cycles per 64 k of 4-bit blocks in two terms at 112 tokens, where the MMAs take 670; in one term 620
// at 160 tokens (320) and 730 at 256 tokens (510).  The model orders plans; it does not predict their times.
Plan make_plan(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int wp, int xp, bool may_split) {
  Plan best = {};
  double best_cost = 1e30;
  const int pairs = ctx->sm_count / 2, kst = wp == 1 || M <= kWideStage ? 2 : 1, nk = (int)((w->nchunks + kst - 1) / kst);
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
  // Operand stages first, but at least two slots of packed weights; what is left goes to the packed ring (few
  // tokens: the weights come from HBM and want tens of KB in flight, and then a stage leaves room for it).
  const size_t stage = (size_t)kst * (wp * kAPlane + xp * (best.bn / 2) * 128), slot = (size_t)slot_bytes_of(w->fmt, kst);
  const size_t room = kSmemBudget - 1024 - 1024;  // alignment, static shared memory
  best.nstages = (int)((room - 2 * slot) / stage);
  const int most = wp == 2 ? 4 : kMaxStages;
  if (best.nstages > most) best.nstages = most;
  best.nslots = (int)((room - best.nstages * stage) / slot);
  best.nslots = (best.nslots < kMaxSlots ? best.nslots : kMaxSlots) & ~1;  // a slot belongs to one dequant set
  best.box_rows = best.bn / 2;
  best.smem = best.nstages * stage + best.nslots * slot + 1024;
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

template <int FMT, int WP, int XP, int KST>
int32_t launch(qeng_ctx* ctx, const qeng_weight* w, const TcParams& p, const Plan& pl, const CUtensorMap& map, cudaStream_t stream) {
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
  p->nstages = pl->nstages; p->nslots = pl->nslots; p->npairs = pl->npairs; p->e = epi;
  p->status = ctx->status;
  return QENG_OK;
}

int32_t qeng_tc::reduce(qeng_ctx* ctx, const TcParams& p, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * p.sk_tiles), (unsigned)(p.bn / 16));
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
  const int64_t parts = gamma == nullptr && M < 2 * ctx->sm_count ? (K + 4 * kPrepThreads - 1) / (4 * kPrepThreads) : 1;
  cfg.gridDim = dim3((unsigned)M, (unsigned)parts);
  cfg.blockDim = dim3(kPrepThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, tc_prep_kernel, x, (int)dtype, (long long)ldx, (int)K, gamma, eps,
                                    reinterpret_cast<__nv_bfloat16*>(out), (long long)(M * K), planes, sums,
                                    (int)((K / 32 + 1) / 2 * 2)));
  return QENG_OK;
}

int32_t qeng_gemm_tc(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, int wp, const qeng_tc_epi& epi, cudaStream_t stream, qeng_scratch* sc) {
  const int xp = x.planes;
  if (w->fmt != QENG_FMT_Q4 && wp == 1) return qeng_fail(ctx, QENG_ERR_SHAPE, "gemm_tc: single bf16 weights are for 4-bit blocks only");
  if (wp == 1 && xp != 1) return qeng_fail(ctx, QENG_ERR_ARG, "gemm_tc: two activation planes need two weight planes");
  Plan pl = make_plan(ctx, w, M, wp, xp, true);
  TcParams p;
  CUtensorMap map;
  if (pl.sk_tiles > 0 && sc == nullptr) sc = qeng_scratch_for(ctx, stream);
  int32_t rc = prepare(ctx, w, x, M, epi, sc, &pl, &p, &map);
  if (rc == QENG_ERR_STATE) {  // no memory for the workspace: whole tiles only
    pl = make_plan(ctx, w, M, wp, xp, false);
    rc = prepare(ctx, w, x, M, epi, sc, &pl, &p, &map);
  }
  if (rc != QENG_OK) return rc;
  if (wp == 1) return launch<QENG_FMT_Q4, 1, 1, 2>(ctx, w, p, pl, map, stream);
#define QENG_TC(F, X) (pl.kst == 2 ? launch<F, 2, X, 2>(ctx, w, p, pl, map, stream) : launch<F, 2, X, 1>(ctx, w, p, pl, map, stream))
  switch (w->fmt) {
    case QENG_FMT_Q4: return xp == 1 ? QENG_TC(QENG_FMT_Q4, 1) : QENG_TC(QENG_FMT_Q4, 2);
    case QENG_FMT_Q8: return xp == 1 ? QENG_TC(QENG_FMT_Q8, 1) : QENG_TC(QENG_FMT_Q8, 2);
    default: return xp == 1 ? QENG_TC(QENG_FMT_K4, 1) : QENG_TC(QENG_FMT_K4, 2);
  }
#undef QENG_TC
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
