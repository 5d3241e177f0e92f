// Quantised matmul of a decode batch (3 to 16 rows of f32 / f16, to 32 of bf16):
//   y[m][n] (f32) = sum over 32-blocks of s[n][block] * (sum_k code[n][k] * x[m][k]), f32 accumulation.
//
// HBM-bound in the ideal: the packed weights are read once.  What bounded the integer path for more than four rows
// was instructions (ten f32 operations per output and block, after five shared loads); here the raw codes are the A
// operand of bf16 MMAs (exact: -8..7, signed bytes, 0..15), the activations the B operand as one bf16 column (bf16
// input) or two (f32, f16: hi and lo, 17 bits) per row, hi and lo in one accumulator, and a block costs two MMAs per
// column tile and one fma per output value.  The contraction order inside a block is the packed one (lane t of a quad
// holds k = 8t .. 8t+7), so A comes from one 128-bit shared load per 64 k and lane, B from one per 32 k and column tile,
// both without conflicts.  With 32 columns the B loads are 32 of 38 shared wavefronts per chunk and bound the kernel
// together with the MMAs (16 rows f32: shared memory busy 63 % of the cycles, the tensor pipe 41 %; 32 rows bf16: 58 and 30).
// 16 rows f32 over 22016 x 4096 30.7 us; 32 rows bf16 over 4096 x 11008 22.0; 8 rows bf16 over 11008 x 4096 11.3 (62, 62 and 15
// with the integer kernel).
//
// Work split: K is cut into `nsl` slices so that a slice of the activations (all columns) stays in shared memory for
// the whole kernel; a CTA owns one slice and every cps-th row tile.  A producer warp streams (tile, slice) units, which
// are contiguous in the packed planes, through a ring with bulk copies; four groups of four warps take the units in
// turn, the warps of a group every fourth chunk.  Partial sums of a unit are parked in shared memory; the CTA meets
// once per `park` units, adds the four warps' parts and writes the slice's sums to a workspace.  A second kernel adds
// the slices in order and runs the epilogue.  (Having the last CTA to arrive at a set of row tiles do that instead left
// a quarter of the chip with all of it: 16 rows over 4096 x 11008 27.5 us against 23.9.)
#include "gemm_tc.cuh"

namespace {
using namespace qeng_tc;

constexpr int kGroups = 4, kGroupWarps = 4, kWarps = kGroups * kGroupWarps, kThreadsR = (kWarps + 1) * 32;
constexpr int kMaxRing = 16;
// Fewer rows: the integer kernel is faster (11008 x 4096: 4 rows f32 10.8 against 11.9 us, bf16: 3 rows 4096 x 4096 7.1 against
// 5.4), except where its shared memory does not hold the activations of all of K, so that it goes over its tiles once per slice
// of K: from 33000 values of f32 or f16 over 8-bit blocks, from 40100 (or a K of 12300) over 4-bit ones.  From 40000 values on,
// over fewer rows of weights than K, the calls come here.  There / here, microseconds, 4-bit and 8-bit: 4 x 11008 over 1024 14.0
// / 7.0, 13.6 / 7.9; over 4096 16.5 / 12.5, 17.9 / 15.1; 3 x 13344 over 4096 18.7 / 13.6, 20.8 / 18.5; 4 x 10016 over 8192 18.6
// / 17.4, 25.7 / 24.4, over 9984 21.4 / 20.4, 30.0 / 27.8.  Below the line 4-bit blocks gain nothing that every shape keeps
// (39936 values over 4096 13.0 / 12.8, 33024 over 4096 12.3 / 11.3, over 8192 17.5 / 18.4, 29952 over 4096 11.7 / 12.5); 8-bit
// ones would gain from 33024 values on (over 4096 16.9 / 13.1, 3 rows 16.2 / 15.0; over 8192 23.6 / 21.0), but over as many rows
// of weights as K neither is ahead (4-bit and 8-bit, 3 x 11008 over 11008 21.2 / 25.3, 29.0 / 31.2, 3 x 13824 over 13824 35.1 /
// 33.0, 43.2 / 50.2).
constexpr int kLeastF32 = 5, kLeastBf16 = 3, kLeastTall = 3;
constexpr int64_t kTallValues = 40000;
// Beyond this many columns the tensor-memory kernel (gemm_tc.cu) takes over.  Here / there, 11008 x 4096, 4-bit: 16 rows bf16 14.2 /
// 21.9 us, 32 rows 21.4 / 22.3, 16 rows f32 (32 columns) 19.7 / 24.6; 8-bit, 32 rows bf16 27.1 / 26.3, 16 rows f32 24.0 / 28.3;
// K-quant, 17 rows bf16 29.7 / 28.6, 32 rows 32.5 / 28.8, 16 rows f32 22.4 / 30.8.  (Over 4096 x 4096 all are faster here.)
constexpr int kMostCols = 32;
constexpr size_t kBudget = 226 * 1024 - 1024;

struct RowsParams {
  const char* qs;
  const char* sc;
  int ntiles, nchunks, K;
  const void* x;           // bf16 planes [XP][M][ldx], brought in as they are, or rows of any type
  int x_dtype, made;
  long long ldx, plane;
  const float* xsum;       // K-quant blocks, planes: [XP][M][nchunks * 2] their block sums
  int M, nsl, cps, slice;  // rows, slices of `slice` chunks, CTAs per slice
  int nring, park;         // ring slots (a multiple of the groups), units parked between meetings
  float* ws;               // [nsl][M][16 * ntiles]
  int32_t* status;
};

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ uint4 ld128(uint32_t a) { return *reinterpret_cast<const uint4*>(__cvta_shared_to_generic((size_t)a)); }
__device__ __forceinline__ uint2 ld64(uint32_t a) { return *reinterpret_cast<const uint2*>(__cvta_shared_to_generic((size_t)a)); }
__device__ __forceinline__ void sts128(uint32_t a, const uint32_t (&w)[4]) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}
__device__ __forceinline__ void stsf(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(a), "f"(v) : "memory"); }
// two f32 values -> bf16 pair and the bf16 pair of what the rounding left
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  hi = u32(h);
  lo = u32(__floats2bfloat162_rn(a - __low2float(h), b - __high2float(h)));
}
__device__ __forceinline__ float ldf(uint32_t a) { return *reinterpret_cast<const float*>(__cvta_shared_to_generic((size_t)a)); }

// (a & b) | c in one instruction: with the constants as literals the compiler spends two, which is 16 of 150 per 64 k
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
struct Consts {
  uint32_t mask, base, sign;  // 4-bit: 0x000f000f, 0x43004300; 8-bit: 0x007f007f, 0x43004300, 0x00800080
};
// pair i (k = 2i, 2i + 1) of a word of 8 codes, as bf16: 4-bit (c - 8), K-quant c
template <int FMT>
__device__ __forceinline__ uint32_t pair4(uint32_t w, int i, const Consts& k) {  // 0x4300 | c is 128 + c
  return u32(__hadd2(bf2(and_or(w >> (4 * i), k.mask, k.base)), bf2(FMT == QENG_FMT_Q4 ? 0xc308c308u : 0xc300c300u)));
}
// 8-bit blocks: a signed byte = (128 + its low 7 bits) - (128, or 256 if the sign bit is set)
__device__ __forceinline__ uint32_t pair8(uint32_t w, int hi, const Consts& k) {
  const uint32_t v = w >> (8 * hi);
  return u32(__hadd2(bf2(and_or(v, k.mask, k.base)), bf2(and_or(v, k.sign, k.base ^ 0x80008000u))));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
// d += a * b on two f32 lanes of a register pair
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float lo_of(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }

// RAW: rows of any type, split into planes here, by every CTA its slice: a call is one launch and one pass through memory less.  f32
// rows over 4-bit blocks, as before / so: 8 over 4096 x 11008 15.5 / 13.5 us, 16 20.9 / 19.4; 8 over 22016 x 4096 23.9 / 21.8; 8
// over 6144 x 4096 12.8 / 10.7; 8-bit blocks 4 to 18 % less.
template <int FMT, int XP, int NT, bool RAW>
// Compiled for more threads than it has: 80 registers leave room on the SM for the CTAs of the second kernel, which are
// then waiting there when this one ends.
__global__ void __launch_bounds__(kThreadsR + 160, 1) gemm_rows_kernel(const RowsParams p) {
  constexpr int kW = Fmt<FMT>::kW, kS = Fmt<FMT>::kS;
  constexpr int kRows = 8 * NT / XP, NR = NT / XP;  // activation rows the tiles hold; accumulators (hi and lo share one)
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kMaxRing], empty[kMaxRing], xbar;
  __shared__ volatile int gave_up;  // a consumer stopped waiting: nobody waits for the producer's copies any more
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int sl = blockIdx.x / p.cps, r0 = blockIdx.x - sl * p.cps;
  const int c0 = sl * p.slice, nc = min(p.slice, p.nchunks - c0);
  const int units = r0 < p.ntiles ? (p.ntiles - r0 + p.cps - 1) / p.cps : 0;
  // shared memory: ring | activation columns (rows of slice * 128 + 64 bytes: two columns of a quarter-warp's load fall
  // into different halves of the banks) | block sums | parked sums
  const uint32_t slot = (uint32_t)p.slice * (kW + kS), xstride = (uint32_t)p.slice * 128u + 64u;
  const uint32_t ring = smem_u32(smem_raw), xs = ring + (uint32_t)p.nring * slot, sums = xs + 8u * NT * xstride;
  const uint32_t sstride = (uint32_t)p.slice * 8u + 16u;
  float* red = reinterpret_cast<float*>(smem_raw + (size_t)p.nring * slot + 8u * NT * xstride + (FMT == QENG_FMT_K4 ? (size_t)XP * kRows * sstride : 0));

  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < p.nring; ++s) {
      mbar_init(smem_u32(full + s), 1);
      mbar_init(smem_u32(empty + s), kGroupWarps);
    }
    mbar_init(smem_u32(&xbar), 1);
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();

  if (warp == kWarps) {
    // ===== producer: one unit = this slice of a row tile, contiguous in both planes ==========================
    if (lane == 0) {
      bool failed = false;
      for (int u = 0; u < units; ++u) {
        const int s = u % p.nring;
        if (!mbar_wait(smem_u32(empty + s), ((uint32_t)(u / p.nring) & 1u) ^ 1u)) { failed = true; break; }
        const uint32_t bar = smem_u32(full + s), dst = ring + (uint32_t)s * slot;
        const size_t at = (size_t)(r0 + u * p.cps) * p.nchunks + c0;
        mbar_expect_tx(bar, (uint32_t)nc * (kW + kS));
        bulk_g2s(dst, p.qs + at * kW, (uint32_t)nc * kW, bar);
        bulk_g2s(dst + (uint32_t)p.slice * kW, p.sc + at * kS, (uint32_t)nc * kS, bar);
      }
      if (failed) atomicExch(p.status, 4);
      if (failed || gave_up) grace();
    }
    return;
  }

  // ===== activations: the columns of this slice ================================================================
  const int kbeg = c0 * 64, kval = min(nc * 64, p.K - kbeg);  // values of K in the slice (a multiple of 32)
  if (!RAW) {
    if (kval < nc * 64)  // the padding block of an odd block count has zero scales: its activations only have to be finite
      for (int i = tid; i < 8 * NT * 4; i += kWarps * 32)
        asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};\n" ::"r"(xs + (uint32_t)(i >> 2) * xstride + (uint32_t)kval * 2u + (uint32_t)(i & 3) * 16u), "r"(0u) : "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (warp == 0) {
      const int cols = XP * p.M;
      if (lane == 0) mbar_expect_tx(smem_u32(&xbar), (uint32_t)(cols * kval * 2));
      __syncwarp();
      for (int c = lane; c < cols; c += 32) {  // column of row m, plane pl: pl * kRows + m
        const int pl = c / p.M, m = c - pl * p.M;
        bulk_g2s(xs + (uint32_t)(pl * kRows + m) * xstride, reinterpret_cast<const __nv_bfloat16*>(p.x) + (size_t)pl * p.plane + (size_t)m * p.ldx + kbeg, (uint32_t)kval * 2u, smem_u32(&xbar));
      }
    }
    if (FMT == QENG_FMT_K4) {
      for (int i = tid; i < XP * p.M * nc * 2; i += kWarps * 32) {
        const int c = i / (nc * 2), b = i - c * nc * 2;  // plane-major: c = plane * M + m
        const float v = p.xsum[(size_t)c * p.nchunks * 2 + c0 * 2 + b];
        asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(sums + (uint32_t)(c / p.M * kRows + c % p.M) * sstride + (uint32_t)b * 4u), "f"(v) : "memory");
      }
    }
  } else {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int ngrp = nc * 8, segs = (ngrp + 31) >> 5;  // groups of 8 k, segments of 32 of them
    const int esz = p.x_dtype == QENG_F32 ? 4 : 2;
    const bool vec = ((reinterpret_cast<uintptr_t>(p.x) | (uintptr_t)(p.ldx * esz)) & 15) == 0;
    const int items = p.M * segs;
    constexpr int kU = 3;  // items of a warp whose loads are on their way together
#pragma unroll 1
    for (int it0 = warp; it0 < items; it0 += kWarps * kU) {
      uint4 raw[kU][2];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int it = it0 + u * kWarps, m = it / segs, k = ((it - m * segs) * 32 + lane) * 8;
        raw[u][0] = raw[u][1] = make_uint4(0u, 0u, 0u, 0u);
        if (it < items && k < kval) {
          const char* src = reinterpret_cast<const char*>(p.x) + ((long long)m * p.ldx + kbeg + k) * esz;
          if (vec) {
            raw[u][0] = *reinterpret_cast<const uint4*>(src);
            if (esz == 4) raw[u][1] = *reinterpret_cast<const uint4*>(src + 16);
          } else {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = esz == 4 ? reinterpret_cast<const uint32_t*>(src)[i] : reinterpret_cast<const uint16_t*>(src)[i];
            if (esz == 4) {
              raw[u][0] = make_uint4(w[0], w[1], w[2], w[3]);
              raw[u][1] = make_uint4(w[4], w[5], w[6], w[7]);
            } else {
              raw[u][0] = make_uint4(w[0] | w[1] << 16, w[2] | w[3] << 16, w[4] | w[5] << 16, w[6] | w[7] << 16);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int it = it0 + u * kWarps;
        if (it >= items) break;
        const int m = it / segs, grp = (it - m * segs) * 32 + lane, k = grp * 8;
        uint32_t hi[4] = {raw[u][0].x, raw[u][0].y, raw[u][0].z, raw[u][0].w}, lo[4] = {0u, 0u, 0u, 0u};
        if (XP == 2) {
          float v[8];
          if (p.x_dtype == QENG_F32) {
            const uint32_t w[8] = {raw[u][0].x, raw[u][0].y, raw[u][0].z, raw[u][0].w, raw[u][1].x, raw[u][1].y, raw[u][1].z, raw[u][1].w};
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(w[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = p.x_dtype == QENG_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&hi[i])) : __bfloat1622float2(bf2(hi[i]));
              v[2 * i] = f.x;
              v[2 * i + 1] = f.y;
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) split2(v[2 * i], v[2 * i + 1], hi[i], lo[i]);
        }
        if (grp < ngrp) {
          sts128(xs + (uint32_t)m * xstride + (uint32_t)k * 2u, hi);
          if (XP == 2) sts128(xs + (uint32_t)(kRows + m) * xstride + (uint32_t)k * 2u, lo);
        }
        if (FMT == QENG_FMT_K4) {  // per block and plane, the sum of the values as stored (the factor of the minimum)
          float q = 0.f, ql = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(bf2(hi[i])), fl = __bfloat1622float2(bf2(lo[i]));
            q += f.x + f.y;
            ql += fl.x + fl.y;
          }
#pragma unroll
          for (int o = 1; o <= 2; o <<= 1) {
            q += __shfl_xor_sync(0xffffffffu, q, o);
            ql += __shfl_xor_sync(0xffffffffu, ql, o);
          }
          if ((lane & 3) == 0 && grp < ngrp) {
            stsf(sums + (uint32_t)m * sstride + (uint32_t)(grp >> 2) * 4u, q);
            if (XP == 2) stsf(sums + (uint32_t)(kRows + m) * sstride + (uint32_t)(grp >> 2) * 4u, ql);
          }
        }
      }
    }
  }
  asm volatile("bar.sync 1, %0;\n" ::"n"(kWarps * 32) : "memory");
  bool failed = !RAW && !mbar_wait(smem_u32(&xbar), 0);

  const int gi = warp / kGroupWarps, wi = warp % kGroupWarps;
  const uint32_t xa = xs + (uint32_t)g * xstride + (uint32_t)t * 16u;  // column g of tile 0, this lane's 8 k
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  const Consts kc = {in_register(FMT == QENG_FMT_Q8 ? 0x007f007fu : 0x000f000fu), in_register(0x43004300u), in_register(0x00800080u)};
  const int rows16 = 16 * p.ntiles;
  for (int u0 = 0; u0 < units; u0 += p.park) {
    const int un = min(p.park, units - u0);
    for (int u = u0 + gi; u < u0 + un; u += kGroups) {  // park is a multiple of the groups: unit u is always group u % 4's
      const int s = u % p.nring;
      if (!failed && !mbar_wait(smem_u32(full + s), (uint32_t)(u / p.nring) & 1u)) failed = true;
      unsigned long long acc[NR][2];  // column tile, row g / g + 8: the lane's two columns
#pragma unroll
      for (int n = 0; n < NR; ++n) acc[n][0] = acc[n][1] = 0ull;
      const uint32_t wb = ring + (uint32_t)s * slot + (uint32_t)lane * 16u, sb = ring + (uint32_t)s * slot + (uint32_t)p.slice * kW;
#pragma unroll 1
      for (int c = wi; c < nc; c += kGroupWarps) {
        const uint4 w0 = ld128(wb + (uint32_t)c * kW);
        uint4 w1;
        if (FMT == QENG_FMT_Q8) w1 = ld128(wb + (uint32_t)c * kW + 512u);
        float sg[2][2], mn[2][2];  // [block][row g, g + 8]
        if (FMT == QENG_FMT_K4) {
          const uint4 d = ld128(sb + (uint32_t)c * kS + (uint32_t)g * 32u), m = ld128(sb + (uint32_t)c * kS + (uint32_t)g * 32u + 16u);
          sg[0][0] = __uint_as_float(d.x); sg[0][1] = __uint_as_float(d.y); sg[1][0] = __uint_as_float(d.z); sg[1][1] = __uint_as_float(d.w);
          mn[0][0] = -__uint_as_float(m.x); mn[0][1] = -__uint_as_float(m.y); mn[1][0] = -__uint_as_float(m.z); mn[1][1] = -__uint_as_float(m.w);
        } else {
          const uint2 s2 = ld64(sb + (uint32_t)c * kS + (uint32_t)g * 8u);
          const float2 e = __half22float2(*reinterpret_cast<const __half2*>(&s2.x)), o = __half22float2(*reinterpret_cast<const __half2*>(&s2.y));
          sg[0][0] = e.x; sg[0][1] = e.y; sg[1][0] = o.x; sg[1][1] = o.y;
        }
        const uint32_t xc = xa + (uint32_t)c * 128u;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          uint32_t a0[4], a1[4];  // K steps (k pairs 0, 1) and (2, 3) of the block
          if (FMT == QENG_FMT_Q8) {
            const uint4 w = b ? w1 : w0;  // bytes 0,4,1,5 of rows g, g + 8; bytes 2,6,3,7
            a0[0] = pair8(w.x, 0, kc); a0[1] = pair8(w.y, 0, kc); a0[2] = pair8(w.z, 0, kc); a0[3] = pair8(w.w, 0, kc);
            a1[0] = pair8(w.x, 1, kc); a1[1] = pair8(w.y, 1, kc); a1[2] = pair8(w.z, 1, kc); a1[3] = pair8(w.w, 1, kc);
          } else {
            const uint32_t u = b ? w0.z : w0.x, v = b ? w0.w : w0.y;
            a0[0] = pair4<FMT>(u, 0, kc); a0[1] = pair4<FMT>(v, 0, kc); a0[2] = pair4<FMT>(u, 1, kc); a0[3] = pair4<FMT>(v, 1, kc);
            a1[0] = pair4<FMT>(u, 2, kc); a1[1] = pair4<FMT>(v, 2, kc); a1[2] = pair4<FMT>(u, 3, kc); a1[3] = pair4<FMT>(v, 3, kc);
          }
          uint4 x[NT];
          float d[NR][4];
#pragma unroll
          for (int n = 0; n < NT; ++n) x[n] = ld128(xc + (uint32_t)(8 * n) * xstride + (uint32_t)b * 64u);
#pragma unroll
          for (int n = 0; n < NR; ++n) mma_bf16(d[n], a0, x[n].x, x[n].y, zero);
#pragma unroll
          for (int n = 0; n < NR; ++n) mma_bf16(d[n], a1, x[n].z, x[n].w, d[n]);
          if (XP == 2) {
#pragma unroll
            for (int n = 0; n < NR; ++n) mma_bf16(d[n], a0, x[NT - NR + n].x, x[NT - NR + n].y, d[n]);
#pragma unroll
            for (int n = 0; n < NR; ++n) mma_bf16(d[n], a1, x[NT - NR + n].z, x[NT - NR + n].w, d[n]);
          }
          const unsigned long long s0 = pack2(sg[b][0], sg[b][0]), s1 = pack2(sg[b][1], sg[b][1]);
#pragma unroll
          for (int n = 0; n < NR; ++n) {
            fma2(acc[n][0], s0, pack2(d[n][0], d[n][1]));
            fma2(acc[n][1], s1, pack2(d[n][2], d[n][3]));
          }
          if (FMT == QENG_FMT_K4) {
            const unsigned long long m0 = pack2(mn[b][0], mn[b][0]), m1 = pack2(mn[b][1], mn[b][1]);
#pragma unroll
            for (int n = 0; n < NR; ++n) {
              const uint32_t sa = sums + (uint32_t)(8 * n + 2 * t) * sstride + (uint32_t)(2 * c + b) * 4u;
              float e0 = ldf(sa), e1 = ldf(sa + sstride);
              if (XP == 2) {
                e0 += ldf(sa + kRows * sstride);
                e1 += ldf(sa + (kRows + 1) * sstride);
              }
              const unsigned long long x2 = pack2(e0, e1);
              fma2(acc[n][0], m0, x2);
              fma2(acc[n][1], m1, x2);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(empty + s));
      // park: [unit][warp of the group][row m][16]
      float* pk = red + (size_t)((u - u0) * kGroupWarps + wi) * (kRows * 16);
#pragma unroll
      for (int n = 0; n < NR; ++n) {
        pk[(8 * n + 2 * t) * 16 + g] = lo_of(acc[n][0]);
        pk[(8 * n + 2 * t + 1) * 16 + g] = hi_of(acc[n][0]);
        pk[(8 * n + 2 * t) * 16 + g + 8] = lo_of(acc[n][1]);
        pk[(8 * n + 2 * t + 1) * 16 + g + 8] = hi_of(acc[n][1]);
      }
    }
    asm volatile("bar.sync 1, %0;\n" ::"n"(kWarps * 32) : "memory");
    // four consecutive weight rows of one (unit, row) per thread
    for (int e = tid; e < un * p.M * 4; e += kWarps * 32) {
      const int u = e / (p.M * 4), q = e - u * (p.M * 4), m = q >> 2, r = (q & 3) * 4;
      const float* src = red + (size_t)u * kGroupWarps * (kRows * 16) + m * 16 + r;
      float4 v = *reinterpret_cast<const float4*>(src);
#pragma unroll
      for (int w = 1; w < kGroupWarps; ++w) {
        const float4 o = *reinterpret_cast<const float4*>(src + w * (kRows * 16));
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
      const int tile = r0 + (u0 + u) * p.cps;
      __stcg(reinterpret_cast<float4*>(p.ws + ((size_t)sl * p.M + m) * rows16 + tile * 16 + r), v);
    }
    if (u0 + p.park < units) asm volatile("bar.sync 1, %0;\n" ::"n"(kWarps * 32) : "memory");
  }
  if (failed) {
    gave_up = 1;
    if (lane == 0) atomicExch(p.status, 4);
    grace();
  }
}

// Sums of the slices and the epilogue.  A warp = 32 weight rows (whole 16-row tiles) x 4 activation rows; up to four
// slices it adds them all, in order.
__global__ void __launch_bounds__(128) rows_finish_kernel(const float* __restrict__ ws, int nsl, int M, int N, const qeng_tc_epi e, int32_t* status) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int lane = threadIdx.x & 31, n = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 32 + lane, m0 = blockIdx.y * 4;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  float f[4] = {0.f, 0.f, 0.f, 0.f};
  if (n < N) {
#pragma unroll 4
    for (int s = 0; s < nsl; ++s) {
      const float* src = ws + ((size_t)s * M + m0) * N + n;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (m0 + i < M) f[i] += __ldcg(src + (size_t)i * N);
    }
  }
  finish<4>(e, N, status, n, m0, M - m0, f, lane);
}
// More than four slices: the four warps of a CTA take every fourth slice of the same 32 weight rows, so that one round
// of loads fetches them all (11 slices in order were three rounds: 16 rows over 4096 x 11008 22.7 us, now 20.1; with four
// slices it is the other way round, 8 rows over 11008 x 4096 11.2 us against 11.7).
__global__ void __launch_bounds__(128) rows_finish_split_kernel(const float* __restrict__ ws, int nsl, int M, int N, const qeng_tc_epi e, int32_t* status) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  __shared__ float part[4][4][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = blockIdx.x * 32 + lane, m0 = blockIdx.y * 4;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  float f[4] = {0.f, 0.f, 0.f, 0.f};
  if (n < N) {
#pragma unroll 3
    for (int s = warp; s < nsl; s += 4) {
      const float* src = ws + ((size_t)s * M + m0) * N + n;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (m0 + i < M) f[i] += __ldcg(src + (size_t)i * N);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) part[warp][i][lane] = f[i];
  __syncthreads();
  if (warp < 2) {
    float v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 2 * warp + i;
      v[i] = (part[0][r][lane] + part[1][r][lane]) + (part[2][r][lane] + part[3][r][lane]);
    }
    finish<2>(e, N, status, n, m0 + 2 * warp, M - m0 - 2 * warp, v, lane);
  }
}

struct RowsPlan {
  bool ok;
  int nt, nsl, cps, slice, nring, park;
  size_t smem;
};

// Slices: the split whose rounds (units per group times chunks per warp) are fewest, with charges for every slice (its
// sums make a round trip through the workspace) and every meeting; a group's ring has two slots at least, or it would
// wait for every refill (four slots for four groups: 31.5 us instead of 26 for 16 rows over 22016 x 4096).
RowsPlan find_plan(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int xp) {
  RowsPlan best = {};
  const int cols = (int)M * xp, sms = ctx->sm_count;
  const int nt = xp == 1 && cols <= 8 ? 1 : cols <= 16 ? 2 : 4;  // two planes: a tile of each at least
  if (cols > kMostCols) return best;
  const int rows = 8 * nt / xp, nch = (int)w->nchunks, ntiles = (int)w->ntiles;
  const size_t per_chunk = (size_t)(chunk_w(w->fmt) + chunk_s(w->fmt)), unit_red = (size_t)kGroupWarps * rows * 16 * 4;
  double best_cost = 1e30;
  for (int nsl = 1; nsl <= nch && nsl <= sms; ++nsl) {
    const int slice = (nch + nsl - 1) / nsl;
    if ((nch + slice - 1) / slice != nsl) continue;
    if (slice < 4 && nsl > 1) break;
    const int cps = sms / nsl < ntiles ? sms / nsl : ntiles;
    const size_t x = (size_t)8 * nt * (slice * 128 + 64) + (w->fmt == QENG_FMT_K4 ? (size_t)xp * rows * (slice * 8 + 16) : 0), slot = slice * per_chunk;
    const int units = (ntiles + cps - 1) / cps, all = (units + kGroups - 1) / kGroups * kGroups;
    int nring = all < 2 * kGroups ? all : 2 * kGroups;
    if (x + kGroups * unit_red + nring * slot > kBudget) continue;
    // parking space for all units if it fits, then more ring, up to about 100 KB
    int park = (int)((kBudget - x - nring * slot) / unit_red) / kGroups * kGroups;
    if (park > all) park = all;
    while (nring + kGroups <= kMaxRing && nring < all && (size_t)nring * slot < 96 * 1024 && x + park * unit_red + (nring + kGroups) * slot <= kBudget)
      nring += kGroups;
    const int meetings = (all + park - 1) / park;
    const double rounds = (double)(all / kGroups) * ((slice + kGroupWarps - 1) / kGroupWarps);
    const double cost = rounds * (1.0 + 0.3 * nt) + 0.25 * nsl * nt + (1.0 + 0.5 * nt) * meetings;
    if (cost < best_cost) {
      best_cost = cost;
      best.ok = true;
      best.nt = nt; best.nsl = nsl; best.cps = cps; best.slice = slice; best.nring = nring; best.park = park;
      best.smem = nring * slot + x + park * unit_red;
    }
  }
  return best;
}

// The search takes a few microseconds of the host: a weight keeps the plans of the last four (rows, planes) it met.
RowsPlan rows_plan(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int xp) {
  std::lock_guard<std::mutex> hold(w->lock);
  for (const auto& e : w->rows_plan)
    if (e[0] == M && e[1] == xp && e[2] == ctx->sm_count) {
      RowsPlan r = {e[3] != 0, e[4], e[5], e[6], e[7], e[8] & 0xff, e[8] >> 8, (size_t)e[9]};
      return r;
    }
  const RowsPlan r = find_plan(ctx, w, M, xp);
  auto& e = w->rows_plan[w->rows_plan_next++ & 3];
  const int v[10] = {(int)M, xp, ctx->sm_count, r.ok ? 1 : 0, r.nt, r.nsl, r.cps, r.slice, r.nring | (r.park << 8), (int)r.smem};
  for (int i = 0; i < 10; ++i) e[i] = v[i];
  return r;
}

template <int FMT, int XP, int NT, bool RAW>
int32_t launch_rows(qeng_ctx* ctx, const RowsParams& p, const RowsPlan& pl, const qeng_tc_epi& e, int N, cudaStream_t stream) {
  static bool configured_on[64] = {};  // the opt-in shared-memory size is set per device
  bool& configured = configured_on[ctx->device & 63];
  if (!configured) {
    QENG_CUDA(ctx, cudaFuncSetAttribute(gemm_rows_kernel<FMT, XP, NT, RAW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBudget));
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pl.nsl * pl.cps));
  cfg.blockDim = dim3(kThreadsR);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, gemm_rows_kernel<FMT, XP, NT, RAW>, p));
  const bool split = p.nsl > 4;
  cfg.gridDim = dim3((unsigned)(split ? (N + 31) / 32 : (N + 127) / 128), (unsigned)((p.M + 3) / 4));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = 0;
  QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, split ? rows_finish_split_kernel : rows_finish_kernel, (const float*)p.ws, p.nsl, p.M, N, e, p.status));
  return QENG_OK;
}

template <int FMT, int XP, bool RAW>
int32_t launch_nt(qeng_ctx* ctx, const RowsParams& p, const RowsPlan& pl, const qeng_tc_epi& e, int N, cudaStream_t stream) {
  switch (pl.nt) {
    case 1: return launch_rows<FMT, 1, 1, RAW>(ctx, p, pl, e, N, stream);  // one plane only
    case 2: return launch_rows<FMT, XP, 2, RAW>(ctx, p, pl, e, N, stream);
    default: return launch_rows<FMT, XP, 4, RAW>(ctx, p, pl, e, N, stream);
  }
}
template <int FMT>
int32_t launch_xp(qeng_ctx* ctx, const RowsParams& p, const RowsPlan& pl, int xp, const qeng_tc_epi& e, int N, cudaStream_t stream) {
  if (p.made) return xp == 1 ? launch_nt<FMT, 1, false>(ctx, p, pl, e, N, stream) : launch_nt<FMT, 2, false>(ctx, p, pl, e, N, stream);
  return xp == 1 ? launch_nt<FMT, 1, true>(ctx, p, pl, e, N, stream) : launch_nt<FMT, 2, true>(ctx, p, pl, e, N, stream);
}

}  // namespace

bool qeng_gemm_rows_planned(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int planes) { return rows_plan(ctx, w, M, planes).ok; }

bool qeng_gemm_rows_fits(const qeng_ctx* ctx, const qeng_weight* w, int64_t M, int planes) {
  const bool tall = w->fmt != QENG_FMT_K4 && w->K > w->N && M * w->K >= kTallValues;
  return M >= (planes == 1 ? kLeastBf16 : tall ? kLeastTall : kLeastF32) && rows_plan(ctx, w, M, planes).ok;
}

static size_t planes_bytes(const qeng_weight* w, int64_t M, int planes) { return ((size_t)planes * M * w->K * 2 + 15) & ~(size_t)15; }

static int32_t rows_call(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int32_t dtype, bool made, const float* xsum, int64_t M, const qeng_tc_epi& epi,
                         cudaStream_t stream, qeng_scratch* sc);

// f32 rows as planes made (and RMS-normalised, if `gamma` is given) by a kernel of its own
int32_t qeng_gemm_rows_prep(qeng_ctx* ctx, const qeng_weight* w, const float* x, int64_t M, int64_t ldx, const float* gamma, float eps,
                            const qeng_tc_epi& epi, cudaStream_t stream) {
  qeng_scratch* sc = qeng_scratch_for(ctx, stream);
  const size_t sum_bytes = w->fmt == QENG_FMT_K4 ? (size_t)2 * M * w->nchunks * 8 : 0;
  int32_t rc = qeng_scratch_grow(ctx, sc, &sc->planes, planes_bytes(w, M, 2) + sum_bytes);
  if (rc != QENG_OK) return rc;
  qeng_tc_x xx;
  xx.data = sc->planes.ptr;
  xx.ld = w->K;
  xx.plane = M * w->K;
  xx.planes = 2;
  float* sums = w->fmt == QENG_FMT_K4 ? reinterpret_cast<float*>(reinterpret_cast<char*>(sc->planes.ptr) + planes_bytes(w, M, 2)) : nullptr;
  rc = qeng_tc_prep(ctx, x, QENG_F32, M, w->K, ldx, gamma, eps, 2, sc->planes.ptr, sums, stream);
  return rc == QENG_OK ? rows_call(ctx, w, xx, QENG_BF16, true, sums, M, epi, stream, sc) : rc;
}

// the working memory of qeng_gemm_rows_prep and qeng_gemm_rows
int32_t qeng_gemm_rows_reserve(qeng_ctx* ctx, const qeng_weight* w, int64_t M, cudaStream_t stream) {
  const RowsPlan pl = rows_plan(ctx, w, M, 2);
  qeng_scratch* sc = qeng_scratch_for(ctx, stream);
  const int32_t rc = qeng_scratch_grow(ctx, sc, &sc->planes, planes_bytes(w, M, 2));
  return rc == QENG_OK ? qeng_scratch_grow(ctx, sc, &sc->part, (size_t)pl.nsl * M * w->N * 4) : rc;
}

// made: x holds bf16 planes, with their block sums in xsum; otherwise rows of any type
static int32_t rows_call(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int32_t dtype, bool made, const float* xsum, int64_t M, const qeng_tc_epi& epi,
                         cudaStream_t stream, qeng_scratch* sc) {
  const RowsPlan pl = rows_plan(ctx, w, M, x.planes);
  if (!pl.ok) return qeng_fail(ctx, QENG_ERR_SHAPE, "gemm_rows: %lld rows over [%lld, %lld] do not fit", (long long)M, (long long)w->N, (long long)w->K);
  if (made && w->fmt == QENG_FMT_K4 && xsum == nullptr) return qeng_fail(ctx, QENG_ERR_ARG, "gemm_rows: K-quant blocks need the block sums of the activations");
  if (sc == nullptr) sc = qeng_scratch_for(ctx, stream);
  const int32_t rc = qeng_scratch_grow(ctx, sc, &sc->part, (size_t)pl.nsl * M * w->N * 4);
  if (rc != QENG_OK) return rc;
  RowsParams p;
  p.qs = reinterpret_cast<const char*>(w->qs); p.sc = reinterpret_cast<const char*>(w->sc);
  p.ntiles = (int)w->ntiles; p.nchunks = (int)w->nchunks; p.K = (int)w->K;
  p.x = x.data; p.x_dtype = dtype; p.made = made; p.ldx = x.ld; p.plane = x.plane; p.xsum = xsum;
  p.M = (int)M; p.nsl = pl.nsl; p.cps = pl.cps; p.slice = pl.slice; p.nring = pl.nring; p.park = pl.park;
  p.ws = reinterpret_cast<float*>(sc->part.ptr);
  p.status = ctx->status;
  switch (w->fmt) {
    case QENG_FMT_Q4: return launch_xp<QENG_FMT_Q4>(ctx, p, pl, x.planes, epi, (int)w->N, stream);
    case QENG_FMT_Q8: return launch_xp<QENG_FMT_Q8>(ctx, p, pl, x.planes, epi, (int)w->N, stream);
    default: return launch_xp<QENG_FMT_K4>(ctx, p, pl, x.planes, epi, (int)w->N, stream);
  }
}

int32_t qeng_gemm_rows(qeng_ctx* ctx, const qeng_weight* w, const qeng_tc_x& x, int64_t M, const qeng_tc_epi& epi, cudaStream_t stream) {
  return rows_call(ctx, w, x, QENG_BF16, true, nullptr, M, epi, stream, nullptr);
}

int32_t qeng_gemm_rows_raw(qeng_ctx* ctx, const qeng_weight* w, const void* x, int32_t dtype, int64_t M, int64_t ldx, const qeng_tc_epi& epi, cudaStream_t stream) {
  qeng_tc_x xx;
  xx.data = x;
  xx.ld = ldx;
  xx.planes = dtype == QENG_BF16 ? 1 : 2;
  const bool made = dtype == QENG_BF16 && w->fmt != QENG_FMT_K4 && ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)(ldx * 2)) & 15) == 0;
  return rows_call(ctx, w, xx, dtype, made, nullptr, M, epi, stream, nullptr);
}
