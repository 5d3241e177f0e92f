// Decode attention (GQA) over a paged f16 KV cache, split over the KV length.
//
// Pool layout: f16 [page][kv head][K|V][16 tokens][128], so the K tile and the
// V tile of one (page, kv head) are 8 KB contiguous.  One CTA serves one
// (sequence, kv head, split).  Each warp looks after the pages it will read: it
// keeps two in flight in shared-memory slots of its own (TMA, 128-byte swizzle,
// completion on an mbarrier) and refills a slot when it has consumed it.  The query heads
// of the group are the eight columns of every MMA, S^T = K Q^T and O^T = V^T P^T,
// so that K and V are the 16-row operands, read with ldmatrix without bank
// conflicts, and no MMA row is wasted on absent heads; P changes its layout with
// movmatrix.  Online softmax (max, sum, out) per query head; warps are merged in shared memory.
// Splits: the CTAs of a thread-block cluster (up to 16) take the pages of a
// sequence round-robin and merge through distributed shared memory (no scratch,
// no atomics); many (sequence, kv head) pairs take fixed page ranges merged
// through a scratch buffer (one per stream, one per capture) by the CTA that arrives last.
//
// HBM-bound: algorithmic bytes = sum_b len_b * kv_heads * 2 * 128 * 2.  With one producer warp for all slots, clusters of
// eight and Q as the (mostly empty) 16-row operand: 1 x 15001 tokens, 8 kv heads 39 us, now 18.5 us (floor 9.4);
// 16 ragged sequences of 512 to 4096 tokens 41 us, now 32.5 us (24.5); 16 of 4096: 74 us, now 48 us (42).
#include <cuda.h>
#include <math.h>

#include "attn_prefill.h"
#include "qeng_internal.h"

namespace {

constexpr int kSlotBytes = 2 * 16 * 128 * 2;
constexpr int kHD = 128;
constexpr int kHDP = kHD + 4;  // row stride of the warps' outputs in shared memory: no bank conflicts
constexpr int kCS = 16;  // largest cluster: CTAs (splits) per sequence and kv head
constexpr int kAW = 4;      // warps per CTA of the fixed splits, three CTAs per SM
constexpr int kAT = kAW * 32;
constexpr int kDepth = 2;  // pages in flight per warp
constexpr int ring_bytes(int warps, int depth) { return warps * depth * kSlotBytes + 1024; }  // and its alignment

__device__ __forceinline__ uint32_t cluster_map(const void* smem_ptr, uint32_t cta_rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(smem_ptr)), "r"(cta_rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
// hardware barrier over all threads of the cluster (every thread of every CTA executes it)
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

struct AttnParams {
  const __half* q;
  const int32_t* table;
  const int32_t* lens;
  float* part_o;   // [B][Hq][S][128]
  float* part_ml;  // [B][Hq][S][2]
  float* out;      // [B][Hq][128]
  int32_t* status;
  int* counters;   // [B][Hkv] arrivals per (sequence, kv head); null = merge in a second kernel
  int pages, Hkv, Hq, grp, max_pages, pps, S;
  float scale, softcap;  // softcap > 0: logits = softcap * tanh(q.k * scale / softcap) (Gemma family)
  int window;            // > 0: only the last `window` tokens of a sequence are attended (sliding window)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up (false) two seconds after the first failed attempt.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
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
// K and V tile of one (page, kv head): 32 rows as two halves of 64 dims, 128-byte swizzled
__device__ __forceinline__ void page_g2s(uint32_t dst, const CUtensorMap* map, int row, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst), "l"(map),
               "r"(0), "r"(row), "r"(0), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
  return d;
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

template <bool kCl, int kW, int kD>
__device__ __forceinline__ void attn_decode_body(const AttnParams& p, const CUtensorMap* kvmap) {
  constexpr int kRing = kD * kW;
  // the output projection that follows may start streaming its weights as CTAs of this kernel retire
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = smem_raw + (1024u - (smem_u32(smem_raw) & 1023u)) % 1024u;  // kRing slots of one page tile
  __shared__ __align__(8) uint64_t full[kRing];
  const int s = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (tid == 0) {
    for (int i = 0; i < kRing; ++i) mbar_init(smem_u32(full + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // Without a window the warp's first 32 page-table entries do not depend on the sequence
  // length: they are asked for together with the length instead of after it (one memory
  // round trip less on the way to the first page).  Entries past the sequence are read (the table
  // row is max_pages long) and never used.
  int pid_cur = -1;
  if (p.window == 0) {
    const int i = warp + kW * lane, idx = kCl ? s + i * p.S : s * p.pps + i;
    if (idx < p.max_pages && (kCl || i < p.pps)) pid_cur = p.table[(size_t)b * p.max_pages + idx];
  }
  __syncthreads();
  // Pages of this CTA, in order: in a cluster the CTAs interleave the pages of the sequence (page =
  // first + cs * i), otherwise a CTA owns the pages [first, first + pps).  With a sliding window the
  // pages that lie entirely before the window are not visited at all.
  const int cs = p.S;  // cluster path: CTAs in the cluster (= gridDim.x)
  const int len = p.lens[b];
  const int npages = min((len + 15) >> 4, p.max_pages);
  const int win0 = p.window > 0 ? max(0, len - p.window) : 0;  // first token inside the window
  const int pg_first = win0 >> 4;
  const int first = kCl ? pg_first + s : pg_first + s * p.pps;
  const int pstep = kCl ? cs : 1;
  const int pend = kCl ? npages : min(npages, pg_first + s * p.pps + p.pps);
  const int n_mine = first < pend ? (pend - first + pstep - 1) / pstep : 0;
  if (!kCl && n_mine == 0) {
    if (p.counters != nullptr && s == 0 && tid < kHD)  // empty sequence: nobody else writes its output
      for (int hh = 0; hh < p.grp; ++hh) p.out[((size_t)b * p.Hq + (size_t)h * p.grp + hh) * kHD + tid] = 0.f;
    return;
  }

  // merge buffers: they live in the ring, which is free once every page of this CTA is consumed
  float (*sm_o)[8][kHDP] = reinterpret_cast<float (*)[8][kHDP]>(ring);                                   // [kW][8][kHDP]
  float (*c_o)[kHD] = reinterpret_cast<float (*)[kHD]>(ring + sizeof(float) * kW * 8 * kHDP);           // [8][kHD]
  float (*sm_m)[8] = reinterpret_cast<float (*)[8]>(ring + sizeof(float) * (kW * 8 * kHDP + 8 * kHD));        // [kW][8]
  float (*sm_l)[8] = sm_m + kW;                                                                        // [kW][8]
  float* c_m = &sm_l[kW][0];                                                                           // [8]
  float* c_l = c_m + 8;                                                                                 // [8]

  // per lane: query heads 2t and 2t + 1 of the group
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float o[8][4];  // O^T: tile j, rows d = 16 j + g and + 8, columns = the lane's two heads
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] = 0.f;

  // Pages warp, warp + kW, ... of the CTA's are this warp's.  It keeps kD of them in flight in slots of its own and refills
  // a slot as soon as it has consumed it: no other warp is involved (one producer warp that looked after every slot of the
  // CTA took 240 ns for each page).  32 page ids at a time, the next 32 asked for one block ahead.
  const int nw = n_mine > warp ? (n_mine - warp + kW - 1) / kW : 0;
  auto page_id = [&](int n) { return n < nw ? p.table[(size_t)b * p.max_pages + first + (warp + kW * n) * pstep] : -1; };
  if (p.window != 0) pid_cur = page_id(lane);
  int pid_next = page_id(32 + lane);
  const uint32_t slots = smem_u32(ring) + (uint32_t)(warp * kD) * kSlotBytes, bars = smem_u32(full + warp * kD);
  auto fetch = [&](int n, int base, int slot) {  // page n of the warp; base: the first page that pid_cur holds
    const int pj = __shfl_sync(0xffffffffu, n - base < 32 ? pid_cur : pid_next, n & 31);
    if (lane == 0) {
      if ((unsigned)pj >= (unsigned)p.pages) {  // malformed page table: record, hand over an empty slot
        atomicExch(p.status, 1);
        mbar_arrive(bars + 8u * slot);
      } else {
        mbar_expect_tx(bars + 8u * slot, kSlotBytes);
        page_g2s(slots + (uint32_t)slot * kSlotBytes, kvmap, (pj * p.Hkv + h) * 32, bars + 8u * slot);
      }
    }
  };
  for (int n = 0; n < kD && n < nw; ++n) fetch(n, 0, n);
  {
    // The group's heads are the 8 columns of every MMA: S^T = K Q^T (rows = 16 tokens), O^T = V^T P^T (rows = 16 dims).
    uint32_t qb[8][2];  // column g = query head h * grp + g (zero columns from grp on)
#pragma unroll
    for (int j = 0; j < 8; ++j) qb[j][0] = qb[j][1] = 0u;
    if (g < p.grp) {
      const uint32_t* qp = reinterpret_cast<const uint32_t*>(p.q + ((size_t)b * p.Hq + (size_t)h * p.grp + g) * kHD);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        qb[j][0] = qp[8 * j + t];
        qb[j][1] = qp[8 * j + 4 + t];
      }
    }
    // ldmatrix rows of this lane: K tokens lane % 16, dims + 8 from lane 16 on; V (transposed) tokens + 8 from lane 16
    // on, dims + 8 in lanes 8-15 and 24-31
    const int krow = lane & 15, kc = lane >> 4, vrow = 16 + (lane & 7) + (lane >> 4) * 8, vc = (lane >> 3) & 1;
    const float sc = p.scale * 1.4426950408889634f;
    auto chunk_at = [](int r, int c) { return (uint32_t)((c >> 3) * 4096 + r * 128 + (((c & 7) ^ (r & 7)) << 4)); };
    auto compute_tile = [&](int pg, uint32_t kv) {
      float sa[2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) sa[0][i] = sa[1][i] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t ka[4];
        ldsm4(kv + chunk_at(krow, 2 * j + kc), ka);
        mma16816(sa[j & 1], ka, qb[j][0], qb[j][1]);
      }
      // scale (optionally soft-capped), log2 domain; lane: tokens g (i < 2) and g + 8, heads 2t and 2t + 1
      const int tok0 = pg * 16;
      const bool edge = tok0 + 16 > len || tok0 < win0;
      float sv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float x = sa[0][i] + sa[1][i];
        if (p.softcap > 0.f) x = p.softcap * tanhf(x * p.scale / p.softcap) * 1.4426950408889634f;
        else x *= sc;
        if (edge) {
          const int tok = tok0 + g + (i >> 1) * 8;
          if (tok >= len || tok < win0) x = -INFINITY;
        }
        sv[i] = x;
      }
      float mx[2] = {fmaxf(sv[0], sv[2]), fmaxf(sv[1], sv[3])}, alpha[2];
#pragma unroll
      for (int o2 = 4; o2 <= 16; o2 <<= 1) {
        mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], o2));
        mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], o2));
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float m_new = fmaxf(m_run[i], mx[i]);  // finite: a listed page holds at least one attended token
        alpha[i] = exp2f(m_run[i] - m_new);
        m_run[i] = m_new;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) sv[i] = exp2f(sv[i] - m_run[i & 1]);
      l_run[0] = l_run[0] * alpha[0] + (sv[0] + sv[2]);
      l_run[1] = l_run[1] * alpha[1] + (sv[1] + sv[3]);
      if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j][0] *= alpha[0]; o[j][1] *= alpha[1];
          o[j][2] *= alpha[0]; o[j][3] *= alpha[1];
        }
      }
      // P as B operand (tokens x heads transposed within the warp), in two f16 terms so no probability precision is lost
      uint32_t hi[2], lo[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        hi[i] = pack_h2(sv[2 * i], sv[2 * i + 1]);
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi[i]));
        lo[i] = transpose8x8(pack_h2(sv[2 * i] - f.x, sv[2 * i + 1] - f.y));
        hi[i] = transpose8x8(hi[i]);
      }
      // V rows that are not attended are zeroed (their probability is 0, but 0 * garbage may be NaN)
      uint32_t keep[2] = {0xffffffffu, 0xffffffffu};
      if (edge) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int tok = tok0 + 8 * i + 2 * t;
          keep[i] = (tok < len && tok >= win0 ? 0xffffu : 0u) | (tok + 1 < len && tok + 1 >= win0 ? 0xffff0000u : 0u);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t va[4];
        ldsm4_t(kv + chunk_at(vrow, 2 * j + vc), va);
        if (edge) {
          va[0] &= keep[0]; va[1] &= keep[0];
          va[2] &= keep[1]; va[3] &= keep[1];
        }
        mma16816(o[j], va, hi[0], hi[1]);
        mma16816(o[j], va, lo[0], lo[1]);
      }
    };
    bool failed = false;
    int slot = 0;
    uint32_t ph = 0;
    for (int n = 0; n < nw; ++n) {
      if ((n & 31) == 0 && n > 0) {
        pid_cur = pid_next;
        pid_next = page_id(n + 32 + lane);
      }
      if (!failed && !mbar_wait(bars + 8u * slot, ph)) failed = true;
      __syncwarp();
      if ((unsigned)__shfl_sync(0xffffffffu, pid_cur, n & 31) < (unsigned)p.pages)
        compute_tile(first + (warp + kW * n) * pstep, slots + (uint32_t)slot * kSlotBytes);
      __syncwarp();
      if (n + kD < nw) fetch(n + kD, n & ~31, slot);
      if (++slot == kD) { slot = 0; ph ^= 1u; }
    }
    if (failed) {
      if (lane == 0) atomicExch(p.status, 4);
      grace();
    }
  }

  // ---- merge the warps of this CTA ------------------------------------------
  __syncthreads();  // every warp is done with the ring: it becomes the merge buffers
  {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int o2 = 4; o2 <= 16; o2 <<= 1) l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], o2);
      const int hh = 2 * t + i;
      if (hh < p.grp) {
        if (g == 0) {
          sm_m[warp][hh] = m_run[i];
          sm_l[warp][hh] = l_run[i];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          sm_o[warp][hh][16 * j + g] = o[j][i];
          sm_o[warp][hh][16 * j + 8 + g] = o[j][2 + i];
        }
      }
    }
  }
  __syncthreads();
  const int ns = kCl ? cs : (npages - pg_first + p.pps - 1) / p.pps;  // splits that hold pages
  const bool direct = !kCl && p.counters != nullptr && ns == 1;  // a single split: no partials needed
  for (int hh = 0; hh < p.grp && tid < kHD; ++hh) {
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kW; ++w) M = fmaxf(M, sm_m[w][hh]);
    float L = 0.f, O = 0.f;
#pragma unroll
    for (int w = 0; w < kW; ++w) {
      const float f = sm_m[w][hh] == -INFINITY ? 0.f : exp2f(sm_m[w][hh] - M);  // a warp without pages
      L += sm_l[w][hh] * f;
      O += sm_o[w][hh][tid] * f;
    }
    if (kCl) {
      c_o[hh][tid] = O;
      if (tid == 0) {
        c_m[hh] = M;
        c_l[hh] = L;
      }
    } else if (direct) {
      p.out[((size_t)b * p.Hq + (size_t)h * p.grp + hh) * kHD + tid] = O / L;
    } else {
      const size_t row = ((size_t)b * p.Hq + (size_t)h * p.grp + hh) * p.S + s;
      __stcg(p.part_o + row * kHD + tid, O);
      if (tid == 0) {
        __stcg(p.part_ml + row * 2, M);
        __stcg(p.part_ml + row * 2 + 1, L);
      }
    }
  }
  if (kCl) {
    // ---- cluster merge: CTA `s` owns 128 / cs dims of every query head and reads the partials of
    // all CTAs of the cluster through distributed shared memory
    if (cs > 1) cluster_sync();
    else __syncthreads();
    const int dper = kHD / cs;
    for (int e = tid; e < p.grp * dper; e += kW * 32) {
      const int hh = e / dper, d = s * dper + e % dper;
      float mr[kCS], lr[kCS], orr[kCS];
#pragma unroll
      for (int r = 0; r < kCS; ++r) {
        mr[r] = -INFINITY;
        lr[r] = orr[r] = 0.f;
        if (r < cs) {
          mr[r] = ld_cluster(cluster_map(&c_m[hh], r));
          lr[r] = ld_cluster(cluster_map(&c_l[hh], r));
          orr[r] = ld_cluster(cluster_map(&c_o[hh][d], r));
        }
      }
      float M = -INFINITY;
#pragma unroll
      for (int r = 0; r < kCS; ++r) M = fmaxf(M, mr[r]);
      float L = 0.f, O = 0.f;
#pragma unroll
      for (int r = 0; r < kCS; ++r) {
        const float f = mr[r] == -INFINITY ? 0.f : exp2f(mr[r] - M);  // a CTA without pages
        L = fmaf(lr[r], f, L);
        O = fmaf(orr[r], f, O);
      }
      p.out[((size_t)b * p.Hq + (size_t)h * p.grp + hh) * kHD + d] = L == 0.f ? 0.f : O / L;  // (an empty sequence; NaN passes)
    }
    if (cs > 1) cluster_sync();  // nobody leaves while a peer may still read its shared memory
    return;
  }
  if (p.counters == nullptr || direct) return;
  // ---- the CTA that completes this (sequence, kv head) merges its splits (no waiting) ----
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(p.counters + b * p.Hkv + h, 1) == ns - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // one warp per query head; lanes first share the (max, sum) pairs of the splits, then each lane
  // merges 4 of the 128 output dims with independent (pipelined) loads
  for (int hh = warp; hh < p.grp; hh += kW) {
    const size_t row0 = ((size_t)b * p.Hq + (size_t)h * p.grp + hh) * p.S;
    float M = -INFINITY;
    for (int s2 = lane; s2 < ns; s2 += 32) M = fmaxf(M, __ldcg(p.part_ml + (row0 + s2) * 2));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float L = 0.f;
    for (int s2 = lane; s2 < ns; s2 += 32) {
      const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + (row0 + s2) * 2));
      L += ml.y * exp2f(ml.x - M);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int s2 = 0; s2 < ns; ++s2) {
      const float f = exp2f(__ldcg(p.part_ml + (row0 + s2) * 2) - M);
      const float4 v = __ldcg(reinterpret_cast<const float4*>(p.part_o + (row0 + s2) * kHD) + lane);
      O.x = fmaf(v.x, f, O.x); O.y = fmaf(v.y, f, O.y); O.z = fmaf(v.z, f, O.z); O.w = fmaf(v.w, f, O.w);
    }
    const float inv = 1.f / L;
    reinterpret_cast<float4*>(p.out + ((size_t)b * p.Hq + (size_t)h * p.grp + hh) * kHD)[lane] =
        make_float4(O.x * inv, O.y * inv, O.z * inv, O.w * inv);
  }
  __syncthreads();
  if (tid == 0) p.counters[b * p.Hkv + h] = 0;  // ready for the next call
}

// three CTAs per SM (<= 136 registers): this path is chosen when there are many pages per SM to cover
__global__ void __launch_bounds__(kAT, 3) attn_decode_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kvmap) {
  attn_decode_body<false, kAW, kDepth>(p, &kvmap);
}

// launched with a cluster dimension of (p.S, 1, 1) = (gridDim.x, 1, 1)
template <int kW, int kD>
__global__ void __launch_bounds__(kW * 32, 1) attn_decode_cluster_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kvmap) {
#ifdef QENG_TRACE
  unsigned long long* rec = nullptr;
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0) rec = qeng_trace_open(p.status, 2);
#endif
  attn_decode_body<true, kW, kD>(p, &kvmap);
#ifdef QENG_TRACE
  if (rec) rec[4] = qeng_trace_now();
#endif
}

__global__ void __launch_bounds__(kHD) attn_combine_kernel(const AttnParams p) {
  const int head = blockIdx.x, b = blockIdx.y, d = threadIdx.x;
  const int len = p.lens[b];
  const int npages = min((len + 15) >> 4, p.max_pages);
  const int pg_first = p.window > 0 ? max(0, len - p.window) >> 4 : 0;
  const int ns = (npages - pg_first + p.pps - 1) / p.pps;
  const size_t row0 = ((size_t)b * p.Hq + head) * p.S;
  float M = -INFINITY;
  for (int s = 0; s < ns; ++s) M = fmaxf(M, p.part_ml[(row0 + s) * 2]);
  float L = 0.f, O = 0.f;
  for (int s = 0; s < ns; ++s) {
    const float f = exp2f(p.part_ml[(row0 + s) * 2] - M);
    L += p.part_ml[(row0 + s) * 2 + 1] * f;
    O += p.part_o[(row0 + s) * kHD + d] * f;
  }
  p.out[((size_t)b * p.Hq + head) * kHD + d] = ns > 0 ? O / L : 0.f;
}

__global__ void kv_append_kernel(__half* pool, const float* k, const float* v, const int32_t* table,
                                 const int32_t* pos, int B, int Hkv, int pages, int max_pages, int32_t* status) {
  const int b = blockIdx.y, h = blockIdx.x, d = threadIdx.x;
  const int ps = pos[b];
  const int pg = ps >> 4;
  if (pg >= max_pages) {
    if (d == 0) atomicExch(status, 2);
    return;
  }
  const int pid = table[(size_t)b * max_pages + pg];
  if ((unsigned)pid >= (unsigned)pages) {
    if (d == 0) atomicExch(status, 1);
    return;
  }
  __half* base = pool + ((size_t)pid * Hkv + h) * (2 * 16 * kHD) + (ps & 15) * kHD + d;
  base[0] = __float2half_rn(k[((size_t)b * Hkv + h) * kHD + d]);
  base[16 * kHD] = __float2half_rn(v[((size_t)b * Hkv + h) * kHD + d]);
}

}  // namespace

static int g_clusters16[64][2];  // per device: clusters of 16 CTAs of 6 and of 4 warps that fit at a time

// opt-in sizes of the cluster kernel with W warps, and how many clusters of 16 the device holds at a time
template <int W>
static int32_t cluster_configure(qeng_ctx* ctx, int* clusters16) {
  auto* fn = attn_decode_cluster_kernel<W, kDepth>;
  QENG_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, ring_bytes(W, kDepth)));
  QENG_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16, 1, 64);
  cfg.blockDim = dim3(W * 32);
  cfg.dynamicSmemBytes = ring_bytes(W, kDepth);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 16;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(clusters16, fn, &cfg) != cudaSuccess) {
    *clusters16 = 0;  // no such clusters here: the launches stay at eight
    (void)cudaGetLastError();
  }
  return QENG_OK;
}

// ---- scratch for the entry point that allocates nothing ---------------------------------
// Some hosts may not allocate device memory once they are running: a runtime that hands the
// engine a fixed memory budget at start-up, or a caller inside a region where the CUDA
// allocator must not be entered (a latency-critical token loop, a process that shares the GPU
// under a hard memory cap).  For them the split partials live in this file-scope array, which
// every GPU that loads the library holds from load to exit.  4 MiB covers
// B * Hq * splits * 130 <= 1048576 floats, e.g. 16 sequences x 32 heads x 15 splits.
constexpr size_t kStaticScratchFloats = (size_t)1 << 20;
static __device__ __align__(256) float g_attn_static_scratch[kStaticScratchFloats];
// In host code the array's name is only a handle: the device address comes from
// cudaGetSymbolAddress, asked once per device with that device current.
constexpr int kMaxDevices = 64;
static float* g_attn_static_addr[kMaxDevices] = {};

constexpr int kMaxAttnCounters = 1 << 16;  // (sequence, kv head) pairs per call

// Splits: enough CTAs to fill the machine several times over, at least one page per warp.
static int pages_per_split(const qeng_ctx* ctx, int64_t B, int64_t Hkv, int64_t max_pages) {
  // the fixed-split kernel keeps three CTAs per SM resident: one full wave of them is the target
  int64_t target = (int64_t)ctx->sm_count * (ctx->attn_ctas_per_sm > 0 ? ctx->attn_ctas_per_sm : 3);
  // splits per (sequence, kv head) that fill the wave without going over it, then equal page ranges for the longest
  // sequence.  (16 sequences of 4096 tokens, 8 kv heads: 3 splits 48 us; 4 splits, a wave and a bit, 55 us.)
  int64_t S = target / (B * Hkv);
  if (S < 1) S = 1;
  int64_t pps = (max_pages + S - 1) / S;
  pps = (pps + kAW - 1) / kAW * kAW;
  if (pps < kAW) pps = kAW;
  if (pps > 128) pps = 128;
  return (int)pps;
}

extern "C" {

int32_t qeng_kv_pool_create(qeng_ctx* ctx, int64_t pages, int64_t kv_heads, int64_t hd, qeng_kv_pool** out) {
  if (!ctx || !out) return qeng_fail(ctx, QENG_ERR_ARG, "kv_pool_create: null argument");
  *out = nullptr;
  if (hd != kHD) return qeng_fail(ctx, QENG_ERR_SHAPE, "kv_pool_create: head_dim must be 128 (got %lld)", (long long)hd);
  if (pages <= 0 || kv_heads <= 0) return qeng_fail(ctx, QENG_ERR_ARG, "kv_pool_create: pages and kv_heads must be positive");
  QENG_CUDA(ctx, cudaSetDevice(ctx->device));
  qeng_kv_pool* p = new qeng_kv_pool();
  p->pages = pages; p->kv_heads = kv_heads; p->hd = hd; p->data = nullptr;
  size_t bytes = (size_t)pages * kv_heads * 2 * 16 * hd * sizeof(__half);
  cudaError_t e = cudaMalloc(&p->data, bytes);
  if (e == cudaSuccess) e = cudaMemset(p->data, 0, bytes);
  if (e != cudaSuccess) {
    if (p->data) cudaFree(p->data);
    delete p;
    return qeng_fail(ctx, QENG_ERR_CUDA, "kv_pool_create: %s", cudaGetErrorString(e));
  }
  *out = p;
  return QENG_OK;
}

int32_t qeng_kv_pool_free(qeng_ctx* ctx, qeng_kv_pool* pool) {
  if (!pool) return QENG_OK;
  if (ctx) cudaSetDevice(ctx->device);
  if (pool->data) cudaFree(pool->data);
  delete pool;
  return QENG_OK;
}

void* qeng_kv_pool_data(const qeng_kv_pool* pool) { return pool ? pool->data : nullptr; }
int64_t qeng_kv_pool_pages(const qeng_kv_pool* pool) { return pool ? pool->pages : 0; }

int32_t qeng_kv_append(qeng_ctx* ctx, qeng_kv_pool* pool, const float* k, const float* v, const int32_t* page_table,
                       int64_t max_pages, const int32_t* pos, int64_t B, void* stream) {
  if (!ctx || !pool || !k || !v || !page_table || !pos) return qeng_fail(ctx, QENG_ERR_ARG, "kv_append: null argument");
  if (B <= 0 || max_pages <= 0) return qeng_fail(ctx, QENG_ERR_ARG, "kv_append: B and max_pages must be positive");
  QENG_ENTER(ctx);
  dim3 grid((unsigned)pool->kv_heads, (unsigned)B);
  kv_append_kernel<<<grid, kHD, 0, (cudaStream_t)stream>>>(pool->data, k, v, page_table, pos, (int)B,
                                                           (int)pool->kv_heads, (int)pool->pages, (int)max_pages,
                                                           ctx->status);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

// opt-in shared memory of the two attention kernels (the page-tile ring), once per device
static int32_t attn_configure(qeng_ctx* ctx) {
  static bool configured_on[64] = {};
  bool& configured = configured_on[ctx->device & 63];
  if (configured) return QENG_OK;
  QENG_CUDA(ctx, cudaFuncSetAttribute(attn_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ring_bytes(kAW, kDepth)));
  int32_t rc = cluster_configure<6>(ctx, &g_clusters16[ctx->device & 63][0]);
  if (rc == QENG_OK) rc = cluster_configure<4>(ctx, &g_clusters16[ctx->device & 63][1]);
  if (rc != QENG_OK) return rc;
  configured = true;
  return QENG_OK;
}

int32_t qeng_attn_decode(qeng_ctx* ctx, const qeng_kv_pool* pool, const uint16_t* q_f16, const int32_t* page_table,
                         int64_t max_pages, const int32_t* lens, int64_t B, int64_t Hq, float scale, float* out,
                         void* stream) {
  return qeng_attn_decode_ex(ctx, pool, q_f16, page_table, max_pages, lens, B, Hq, scale, 0.f, 0, out, stream);
}

int32_t qeng_attn_decode_ex(qeng_ctx* ctx, const qeng_kv_pool* pool, const uint16_t* q_f16, const int32_t* page_table,
                            int64_t max_pages, const int32_t* lens, int64_t B, int64_t Hq, float scale, float softcap,
                            int32_t window, float* out, void* stream) {
  if (!ctx || !pool || !q_f16 || !page_table || !lens || !out) return qeng_fail(ctx, QENG_ERR_ARG, "attn_decode: null argument");
  if (B <= 0 || max_pages <= 0 || Hq <= 0) return qeng_fail(ctx, QENG_ERR_ARG, "attn_decode: B, Hq, max_pages must be positive");
  if (softcap < 0.f || window < 0) return qeng_fail(ctx, QENG_ERR_ARG, "attn_decode: softcap and window must not be negative");
  if (Hq % pool->kv_heads != 0 || Hq / pool->kv_heads > 8)
    return qeng_fail(ctx, QENG_ERR_SHAPE, "attn_decode: query heads per kv head must divide evenly and be <= 8");
  if (((reinterpret_cast<uintptr_t>(q_f16) | reinterpret_cast<uintptr_t>(out)) & 15) != 0)
    return qeng_fail(ctx, QENG_ERR_ALIGN, "attn_decode: q and out must be 16-byte aligned");
  QENG_ENTER(ctx);
  int32_t rc0 = attn_configure(ctx);
  if (rc0 != QENG_OK) return rc0;
  AttnParams p;
  p.q = reinterpret_cast<const __half*>(q_f16);
  p.table = page_table; p.lens = lens; p.out = out; p.status = ctx->status;
  p.pages = (int)pool->pages; p.Hkv = (int)pool->kv_heads; p.Hq = (int)Hq; p.grp = (int)(Hq / pool->kv_heads);
  p.max_pages = (int)max_pages;
  p.scale = scale; p.softcap = softcap; p.window = window;
  CUtensorMap map;
  int32_t rc1 = qeng_kv_map(ctx, pool->data, pool->pages * pool->kv_heads * 32, &map);
  if (rc1 != QENG_OK) return rc1;
  // Cluster path: as many CTAs per (sequence, kv head) as keep the grid within two CTAs per SM, sixteen where the device
  // holds all the clusters of sixteen at a time (of 6 warps, else of 4).  Below four CTAs per pair the fixed splits are
  // as fast on long caches and faster on short ones (16 x 64 tokens: 4.8 against 7.0 us).
  const int64_t pairs = B * pool->kv_heads;
  const int* clusters16 = g_clusters16[ctx->device & 63];
  int cs = 8, warps = 6;
  if (pairs <= clusters16[0]) {
    cs = 16;
  } else if (pairs <= clusters16[1]) {
    cs = 16;
    warps = 4;
  }
  while (cs > 1 && pairs * cs > 2 * (int64_t)ctx->sm_count) cs >>= 1;
  bool cluster = ctx->attn_cluster && cs >= 4;
  qeng_scratch* sc = nullptr;
  if (!cluster) {
    p.pps = pages_per_split(ctx, B, pool->kv_heads, max_pages);
    p.S = (int)((max_pages + p.pps - 1) / p.pps);
    if (pairs > kMaxAttnCounters)
      return qeng_fail(ctx, QENG_ERR_SHAPE, "attn: B * kv_heads = %lld exceeds %d", (long long)pairs, kMaxAttnCounters);
    // arrival counters first (fixed place for every shape; they start at zero and return to it), partials behind them
    sc = qeng_scratch_for(ctx, (cudaStream_t)stream);
    const size_t need = (size_t)kMaxAttnCounters * sizeof(int) + (size_t)B * Hq * p.S * (kHD + 2) * sizeof(float);
    const int32_t rc = qeng_scratch_grow(ctx, sc, &sc->attn, need, true);
    if (rc != QENG_OK && (!ctx->attn_cluster || !ctx->no_memory)) return rc;
    cluster = rc != QENG_OK;  // no memory for the partials: clusters need none
  }
  if (cluster) {
    p.pps = 0; p.S = cs; p.counters = nullptr; p.part_o = nullptr; p.part_ml = nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cs, (unsigned)p.Hkv, (unsigned)B);
    cfg.blockDim = dim3((unsigned)warps * 32);
    cfg.dynamicSmemBytes = ring_bytes(warps, kDepth);
    cfg.stream = (cudaStream_t)stream;
    // (launched with programmatic serialisation as well, a one-sequence decode step got 2 % slower: the CTAs that wait
    // keep shared memory from the matmul in front)
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    QENG_CUDA(ctx, cudaLaunchKernelEx(&cfg, warps == 6 ? attn_decode_cluster_kernel<6, kDepth> : attn_decode_cluster_kernel<4, kDepth>, p, map));
    return QENG_OK;
  }
  p.counters = reinterpret_cast<int*>(sc->attn.ptr);
  p.part_o = reinterpret_cast<float*>(sc->attn.ptr) + kMaxAttnCounters;
  p.part_ml = p.part_o + (size_t)B * Hq * p.S * kHD;
  dim3 grid((unsigned)p.S, (unsigned)p.Hkv, (unsigned)B);
  attn_decode_kernel<<<grid, kAT, ring_bytes(kAW, kDepth), (cudaStream_t)stream>>>(p, map);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

int32_t qeng_attn_decode_noalloc(qeng_ctx* ctx, const qeng_kv_pool* pool, const uint16_t* q_f16,
                                 const int32_t* page_table, int64_t max_pages, const int32_t* lens, int64_t B,
                                 int64_t Hq, float scale, float* out, void* stream) {
  if (!ctx || !pool || !q_f16 || !page_table || !lens || !out)
    return qeng_fail(ctx, QENG_ERR_ARG, "attn_decode_noalloc: null argument");
  if (B <= 0 || max_pages <= 0 || Hq <= 0)
    return qeng_fail(ctx, QENG_ERR_ARG, "attn_decode_noalloc: B, Hq, max_pages must be positive");
  if (Hq % pool->kv_heads != 0 || Hq / pool->kv_heads > 8)
    return qeng_fail(ctx, QENG_ERR_SHAPE, "attn_decode_noalloc: query heads per kv head must divide evenly and be <= 8");
  if ((reinterpret_cast<uintptr_t>(q_f16) & 15) != 0)
    return qeng_fail(ctx, QENG_ERR_ALIGN, "attn_decode_noalloc: q must be 16-byte aligned");
  if (ctx->device < 0 || ctx->device >= kMaxDevices)
    return qeng_fail(ctx, QENG_ERR_ARG, "attn_decode_noalloc: device index %d outside 0..%d", ctx->device, kMaxDevices - 1);
  QENG_ENTER(ctx);
  AttnParams p;
  p.pps = pages_per_split(ctx, B, pool->kv_heads, max_pages);
  p.S = (int)((max_pages + p.pps - 1) / p.pps);
  const size_t need = (size_t)B * Hq * p.S * (kHD + 2);
  if (need > kStaticScratchFloats)
    return qeng_fail(ctx, QENG_ERR_SHAPE,
                     "attn_decode_noalloc: B*Hq*splits*130 = %zu floats exceeds the built-in scratch of %zu floats "
                     "(B=%lld Hq=%lld splits=%d); use qeng_attn_decode",
                     need, kStaticScratchFloats, (long long)B, (long long)Hq, p.S);
  // set-up, once per device: resolve the array's device address with that device current
  if (!g_attn_static_addr[ctx->device]) {
    QENG_CUDA(ctx, cudaSetDevice(ctx->device));
    float* addr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&addr), g_attn_static_scratch);
    if (e != cudaSuccess || !addr)
      return qeng_fail(ctx, QENG_ERR_CUDA, "attn_decode_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    g_attn_static_addr[ctx->device] = addr;
  }
  float* scratch = g_attn_static_addr[ctx->device];
  p.q = reinterpret_cast<const __half*>(q_f16);
  p.table = page_table; p.lens = lens; p.out = out; p.status = ctx->status;
  p.pages = (int)pool->pages; p.Hkv = (int)pool->kv_heads; p.Hq = (int)Hq; p.grp = (int)(Hq / pool->kv_heads);
  p.max_pages = (int)max_pages;
  p.scale = scale; p.softcap = 0.f; p.window = 0;
  {
    int32_t rc0 = attn_configure(ctx);
    if (rc0 != QENG_OK) return rc0;
  }
  CUtensorMap map;
  {
    int32_t rc0 = qeng_kv_map(ctx, pool->data, pool->pages * pool->kv_heads * 32, &map);
    if (rc0 != QENG_OK) return rc0;
  }
  // every partial that the merge reads is written by this call first: nothing has to start at zero
  p.counters = nullptr;  // merge in a second kernel
  p.part_o = scratch;
  p.part_ml = scratch + (size_t)B * Hq * p.S * kHD;
  dim3 grid((unsigned)p.S, (unsigned)p.Hkv, (unsigned)B);
  attn_decode_kernel<<<grid, kAT, ring_bytes(kAW, kDepth), (cudaStream_t)stream>>>(p, map);
  QENG_LAUNCH_CHECK(ctx);
  dim3 grid2((unsigned)Hq, (unsigned)B);
  attn_combine_kernel<<<grid2, kHD, 0, (cudaStream_t)stream>>>(p);
  QENG_LAUNCH_CHECK(ctx);
  return QENG_OK;
}

}  // extern "C"
