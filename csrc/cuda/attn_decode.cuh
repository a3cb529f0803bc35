// Decode body of the grouped-query attention kernel: every row is one query token of its own sequence (head dim 128, at
// most 8 query heads per kv head), over the paged bf16 or e4m3 cache.
//
// A decode step reads each cached key and value once and does 2 x group multiply-adds per element, so it is bound by the
// stream from HBM.  The 128-lane tile form pays for its shape there: four heads fill 4 of 128 lanes, items of whole
// sequences leave SMs idle when lengths differ (170 us for 64 sequences of 512 to 4352 tokens, 98 us of traffic), and the
// e4m3 cache has to be rewritten as bf16 tiles in shared memory (268 us for half the traffic).  Here:
//   * all (row, kv head, page) triples of the step form one line, cut into equal pieces, one per CTA: every SM streams the
//     same number of pages.  A (row, kv head) that is cut leaves f32 partials; the CTA that finishes it last folds them.
//   * one warp feeds a ring of pages (TMA; the e4m3 scales by 4-byte cp.async), eight warps consume: four share a page, 16
//     tokens each, so two pages are in work at a time.  S = Q K^T and O += P V are m16n8k16 warp MMAs with the heads as
//     rows; every warp keeps its own running maximum, sum and O, merged through shared memory when a piece ends.
//   * e4m3 elements become bf16 in registers: the byte s.eeee.mmm placed as s.0000eeee.mmm0000 is value * 2^-120, four
//     integer instructions per pair; key scales multiply S, value scales P, and the powers of two go with them.  The k index
//     of an MMA may be any permutation as long as both operands agree, so a lane takes 16 consecutive bytes of a row.
// The rates of mma.sync suffice by far (64 of 356 clocks per 16 tokens and SM).
#pragma once
#include <cuda_bf16.h>

#include "ptx.cuh"

namespace plow {

constexpr int kDecThreads = 320;          // 8 consumer warps, the producer warp, one idle
constexpr int kDecMaxCtas = 160;
constexpr int kDecMaxGroup = 8;
constexpr int kDecMaxRows = 256;
constexpr int kDecPartial = kDecMaxGroup * 130;      // floats of a partial: [head][128] O, then [head] m, [head] l

// Scratch of a call, in 4-byte words: plan (8), prefix of pages [rows + 1], arrivals [rows * nkv], partials [2 per CTA].
struct DecScratch {
  int* plan;            // [0]: 1 = this call is a decode step; [1]: pages
  int* prefix;
  int* arrived;
  float* partial;
  __host__ __device__ DecScratch(void* base, int rows, int nkv) {
    plan = static_cast<int*>(base);
    prefix = plan + 8;
    arrived = prefix + rows + 1;
    partial = reinterpret_cast<float*>(arrived + rows * nkv);
  }
  static int64_t bytes(int rows, int nkv) {
    return 4ll * (8 + rows + 1 + static_cast<int64_t>(rows) * nkv + 2ll * kDecMaxCtas * kDecPartial);
  }
};

struct DecArgs {
  void* scratch;
  const __nv_bfloat16* q;
  const int* page_table;
  const int* pos;
  const int* seq;
  const float* kv_scale;
  __nv_bfloat16* out;
  int* status;
  int rows, nq, nkv, group, max_pages, window;
  float scale_log2e;
};

template <bool KV8> struct DecCfg {
  // Even: stage s then always belongs to the same four warps.  With an odd ring a group would wait for every other phase of a
  // stage only, and a parity wait cannot tell a phase from the one two before it.
  static constexpr int kStages = KV8 ? 8 : 4;
  static_assert(kStages % 2 == 0, "a stage belongs to one group of warps");
  static constexpr int kTile = KV8 ? 8192 : 16384;               // one page of keys or values of a head
  static constexpr int kStage = 2 * kTile + (KV8 ? 512 : 0);     // + 64 key and 64 value scales
  // ring, control, then the merge area: [8 warps][heads][132] f32
  static constexpr int kStageStride = (kStage + 1023) / 1024 * 1024;
  static constexpr int kRing = kStages * kStageStride;
  static constexpr int smem(int group) { return 1024 + kRing + 4096 + 8 * group * 132 * 4; }
};

__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float dec_ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// two e4m3 bytes in the high bytes of two 16-bit lanes -> bf16x2 of value * 2^-120
__device__ __forceinline__ uint32_t e4m3_lanes_to_bf16(uint32_t x) { return (x & 0x80008000u) | ((x >> 4) & 0x07f007f0u); }

template <bool KV8>
__device__ void gqa_decode_body(const DecArgs& a, const CUtensorMap* tm_k, const CUtensorMap* tm_v) {
  using Cfg = DecCfg<KV8>;
  constexpr int kS = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* ctrl = ring + Cfg::kRing;
  uint64_t* full = reinterpret_cast<uint64_t*>(ctrl);        // [kS]
  uint64_t* empty = full + kS;                               // [kS]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kS);
  int* last_flag = const_cast<int*>(abort_flag) + 1;
  int* prefix = reinterpret_cast<int*>(ctrl + 512);          // [rows + 1]
  float* area = reinterpret_cast<float*>(ctrl + 4096);       // [8][group][132]: O, m, l
  const DecScratch sc(a.scratch, a.rows, a.nkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = sc.plan[1];
  const int G = min(static_cast<int>(gridDim.x), T);
  if (static_cast<int>(blockIdx.x) >= G) return;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kS; ++s) { mbar_init(&full[s], KV8 ? 33 : 1); mbar_init(&empty[s], 4); }
    *abort_flag = 0;
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i <= a.rows; i += kDecThreads) prefix[i] = sc.prefix[i];
  __syncthreads();
  const int p0 = static_cast<int>(static_cast<long long>(T) * blockIdx.x / G), p1 = static_cast<int>(static_cast<long long>(T) * (blockIdx.x + 1) / G);
  // the piece that starts at page p of the line: its row, kv head, first page within the sequence's span, length
  struct Piece { int row, kvh, first, n, pages, lo_page, hi, lo; };
  auto piece_at = [&](int p) -> Piece {
    int x = 0, y = a.rows;                                   // last row whose prefix is <= p (empty rows never qualify)
    while (y - x > 1) { const int m = (x + y) >> 1; if (prefix[m] <= p) x = m; else y = m; }
    Piece c;
    c.row = x;
    c.hi = a.pos[x];
    c.lo = a.window > 0 ? max(0, c.hi - a.window + 1) : 0;
    c.lo_page = c.lo / 64;
    c.pages = c.hi / 64 - c.lo_page + 1;
    const int o = p - prefix[x];
    c.kvh = o / c.pages;
    c.first = o % c.pages;
    c.n = min(c.pages - c.first, p1 - p);
    return c;
  };

  if (warp == 8) {
    // ------------------------------------------------------------------ producer
    uint32_t k = 0;
    bool ok = true;
    for (int p = p0; ok && p < p1;) {
      const Piece c = piece_at(p);
      const int* pt = a.page_table + static_cast<size_t>(a.seq[c.row]) * a.max_pages + c.lo_page + c.first;
      // a lane holds the page number of one of the next 32 pages
      for (int i0 = 0; ok && i0 < c.n; i0 += 32) {
        const int mine = i0 + lane < c.n ? pt[i0 + lane] : 0;
        for (int i = i0; i < min(c.n, i0 + 32); ++i, ++k) {
          const int page = __shfl_sync(0xffffffffu, mine, i - i0);
          const int s = k % kS;
          if (!mbar_wait(&empty[s], ((k / kS) & 1) ^ 1, abort_flag)) {
            *abort_flag = 1; atomicCAS(a.status, 0, PLOW_ERR_STAGE_WAIT | kTagGqa); ok = false; break;
          }
          uint8_t* st = ring + s * Cfg::kStageStride;
          if (lane == 0) {
            mbar_expect_tx(&full[s], 2 * Cfg::kTile);
            if constexpr (KV8) {
              tma_load_3d(st, tm_k, 0, c.kvh, page * 64, &full[s]);
              tma_load_3d(st + Cfg::kTile, tm_v, 0, c.kvh, page * 64, &full[s]);
            } else {
              tma_load_3d(st, tm_k, 0, c.kvh, page * 64, &full[s]);
              tma_load_3d(st + 8192, tm_k, 64, c.kvh, page * 64, &full[s]);
              tma_load_3d(st + Cfg::kTile, tm_v, 0, c.kvh, page * 64, &full[s]);
              tma_load_3d(st + Cfg::kTile + 8192, tm_v, 64, c.kvh, page * 64, &full[s]);
            }
          }
          if constexpr (KV8) {
            // scales of the 64 tokens: key scales, then value scales
            const float* src = a.kv_scale + static_cast<size_t>(page) * 64 * 2 * a.nkv + c.kvh;
            const uint32_t dst = smem_u32(st + 2 * Cfg::kTile);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int e = u * 32 + lane;
              const float* g = src + static_cast<size_t>(e & 63) * 2 * a.nkv + (e >= 64 ? a.nkv : 0);
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + e * 4), "l"(g) : "memory");
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s])) : "memory");
          }
        }
      }
      p += c.n;
    }
    if (KV8) asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp < 8) {
    // ------------------------------------------------------------------ consumers
    const int duo = warp >> 2, tok0 = (warp & 3) * 16;       // which of two pages in turn, which 16 of its tokens
    const int g = lane >> 2, c4 = lane & 3;
    uint32_t k0 = 0;                                         // pages of the pieces before
    bool ok = true;
    for (int p = p0; p < p1;) {
      const Piece c = piece_at(p);
      // Q fragments: MMA rows 0 .. 7 are the heads of this kv head, rows 8 .. 15 stay zero.  k-step s covers dims 16 s + {2 c4, 2 c4 + 1, + 8, + 9};
      // for e4m3 dims 64 (s / 4) + 16 c4 + 4 (s % 4) + {0, 1, 2, 3} in the same places
      uint32_t qa[8][4];
      const __nv_bfloat16* qr = a.q + (static_cast<size_t>(c.row) * a.nq + c.kvh * a.group) * 128;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int d0 = KV8 ? 64 * (s >> 2) + 16 * c4 + 4 * (s & 3) : 16 * s + 2 * c4, d1 = KV8 ? d0 + 2 : d0 + 8;
        qa[s][0] = g < a.group ? *reinterpret_cast<const uint32_t*>(qr + g * 128 + d0) : 0u;
        qa[s][1] = 0u;
        qa[s][2] = g < a.group ? *reinterpret_cast<const uint32_t*>(qr + g * 128 + d1) : 0u;
        qa[s][3] = 0u;
      }
      float o[16][4];
#pragma unroll
      for (int n = 0; n < 16; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[n][j] = 0.f;
      float m = -1e30f, l = 0.f;
      for (int i = (duo ^ (k0 & 1)); ok && i < c.n; i += 2) {
        const uint32_t k = k0 + i;
        const int s = k % kS;
        if (!mbar_wait(&full[s], (k / kS) & 1, abort_flag)) { *abort_flag = 1; atomicCAS(a.status, 0, PLOW_ERR_TMA_WAIT | kTagGqa); ok = false; break; }
        const uint8_t* st = ring + s * Cfg::kStageStride;
        float sc4[2][4];                                     // S of tokens tok0 + 8 t + 2 c4 + {0, 1}, head g in [0], [1]
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int j = 0; j < 4; ++j) sc4[t][j] = 0.f;
        if constexpr (KV8) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int row = tok0 + 8 * t + g;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint4 w = *reinterpret_cast<const uint4*>(st + row * 128 + ((4 * h + c4) ^ (row & 7)) * 16);
              const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
              for (int u = 0; u < 4; ++u)
                mma_bf16(sc4[t], qa[4 * h + u], e4m3_lanes_to_bf16(__byte_perm(ww[u], 0, 0x1404)), e4m3_lanes_to_bf16(__byte_perm(ww[u], 0, 0x3424)));
            }
          }
        } else {
          // 8x8 blocks of an ldmatrix.x4: tokens 8 t .. + 7, dims 16 s .. + 15 and the next 16
          const uint32_t kb = smem_u32(st);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int row = tok0 + 8 * t + (lane & 7);
#pragma unroll
            for (int s2 = 0; s2 < 4; ++s2) {
              const int chunk = 4 * s2 + (lane >> 3);        // 16-byte chunk of the 256-byte row
              uint32_t b[4];
              ldmatrix4(kb + (chunk >> 3) * 8192 + row * 128 + ((chunk & 7) ^ (row & 7)) * 16, b);
              mma_bf16(sc4[t], qa[2 * s2], b[0], b[1]);
              mma_bf16(sc4[t], qa[2 * s2 + 1], b[2], b[3]);
            }
          }
        }
        float vs[4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int tok = tok0 + 8 * t + 2 * c4;
          float f0 = a.scale_log2e, f1 = a.scale_log2e;
          if constexpr (KV8) {
            const float* scs = reinterpret_cast<const float*>(st + 2 * Cfg::kTile);
            const float2 ks = *reinterpret_cast<const float2*>(scs + tok), v2 = *reinterpret_cast<const float2*>(scs + 64 + tok);
            const float top = a.scale_log2e * 0x1p120f;
            f0 = fmaxf(fminf(ks.x * top, 3.0e38f), -3.0e38f); f1 = fmaxf(fminf(ks.y * top, 3.0e38f), -3.0e38f);
            vs[2 * t] = fminf(v2.x * 0x1p60f, 3.0e38f); vs[2 * t + 1] = fminf(v2.y * 0x1p60f, 3.0e38f);
          }
          sc4[t][0] *= f0; sc4[t][1] *= f1;
        }
        const int t0 = (c.lo_page + c.first + i) * 64 + tok0;
        if (t0 < c.lo || t0 + 15 > c.hi) {
#pragma unroll
          for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int tok = t0 + 8 * t + 2 * c4 + j;
              if (tok < c.lo || tok > c.hi) sc4[t][j] = -INFINITY;
            }
        }
        // running maximum per head, moved only when exceeded by more than 2^7 (P then stays below that)
        float mx = fmaxf(fmaxf(sc4[0][0], sc4[0][1]), fmaxf(sc4[1][0], sc4[1][1]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const bool up = mx > m + 7.0f;
        if (__any_sync(0xffffffffu, up)) {
          const float n = up ? mx : m, f = dec_ex2(m - n);
          l *= f;
          m = n;
#pragma unroll
          for (int j = 0; j < 16; ++j) { o[j][0] *= f; o[j][1] *= f; }
        }
        // P: the accumulator layout of S is the A layout of the next MMA (k = token)
        uint32_t pa[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          float e0 = dec_ex2(sc4[t][0] - m), e1 = dec_ex2(sc4[t][1] - m);
          l += e0 + e1;
          if constexpr (KV8) { e0 *= vs[2 * t]; e1 *= vs[2 * t + 1]; }
          const __nv_bfloat162 h0 = __floats2bfloat162_rn(e0, e1);
          pa[2 * t] = *reinterpret_cast<const uint32_t*>(&h0);
        }
        const uint8_t* vt = st + Cfg::kTile;
        if constexpr (KV8) {
          // a lane takes 16 bytes (dims 16 g .. + 15) of the four tokens of its k indices; column g of n-tile n is dim 16 g + n
          uint32_t w[4][4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int row = tok0 + 2 * c4 + (u & 1) + 8 * (u >> 1);
            const uint4 x = *reinterpret_cast<const uint4*>(vt + row * 128 + (g ^ (row & 7)) * 16);
            w[u][0] = x.x; w[u][1] = x.y; w[u][2] = x.z; w[u][3] = x.w;
          }
#pragma unroll
          for (int n = 0; n < 16; ++n) {
            // byte n of tokens (2 c4, 2 c4 + 1) and (+ 8, + 9) into the high bytes of the two lanes (the low bytes are cut
            // off by the mask, whatever they hold)
            const uint32_t sel = ((n & 3) << 4) | ((4 + (n & 3)) << 12);
            const uint32_t b0 = __byte_perm(w[0][n >> 2], w[1][n >> 2], sel), b1 = __byte_perm(w[2][n >> 2], w[3][n >> 2], sel);
            mma_bf16(o[n], pa, e4m3_lanes_to_bf16(b0), e4m3_lanes_to_bf16(b1));
          }
        } else {
          const uint32_t vb = smem_u32(vt);
          const int row = tok0 + (lane & 15);
#pragma unroll
          for (int n = 0; n < 8; ++n) {
            // 8x8 blocks: tokens 0 .. 7 and 8 .. 15 of dims 16 n .. + 7, then of dims 16 n + 8 .. + 15
            const int chunk = 2 * n + (lane >> 4);
            uint32_t b[4];
            ldmatrix4_trans(vb + (chunk >> 3) * 8192 + row * 128 + ((chunk & 7) ^ (row & 7)) * 16, b);
            mma_bf16(o[2 * n], pa, b[0], b[1]);
            mma_bf16(o[2 * n + 1], pa, b[2], b[3]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
      }
      k0 += c.n;
      p += c.n;
      // ---- the piece is done: merge the eight warps (each holds a partial over its tokens)
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
      if (g < a.group) {
        float* dst = area + (warp * a.group + g) * 132;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          // dims of columns 2 c4 and 2 c4 + 1 of n-tile n
          const int d0 = KV8 ? 32 * c4 + n : 8 * n + 2 * c4, d1 = KV8 ? 32 * c4 + 16 + n : d0 + 1;
          dst[d0] = o[n][0];
          dst[d1] = o[n][1];
        }
        if (c4 == 0) { dst[128] = m; dst[129] = l; }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const int u0 = prefix[c.row] + c.kvh * c.pages;                              // the line's pages of this (row, kv head)
      const int b0 = static_cast<int>((static_cast<long long>(u0 + 1) * G - 1) / T), b1 = static_cast<int>((static_cast<long long>(u0 + c.pages) * G - 1) / T);
      const bool whole = b0 == b1;
      const bool is_first = p - c.n == p0;
      float* part = sc.partial + (static_cast<size_t>(blockIdx.x) * 2 + (is_first ? 0 : 1)) * kDecPartial;
      __nv_bfloat16* orow = a.out + (static_cast<size_t>(c.row) * a.nq + c.kvh * a.group) * 128;
      constexpr float kOut = KV8 ? 0x1p60f : 1.0f;                                // the e4m3 accumulator carries 2^-60
      for (int e = threadIdx.x; e < a.group * 128; e += 256) {
        const int head = e >> 7, d = e & 127;
        const float* src = area + head * 132;
        const int stride = a.group * 132;
        float top = -1e30f;
#pragma unroll
        for (int w = 0; w < 8; ++w) top = fmaxf(top, src[w * stride + 128]);
        float acc = 0.f, sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          const float f = dec_ex2(src[w * stride + 128] - top);
          acc += f * src[w * stride + d];
          sum += f * src[w * stride + 129];
        }
        acc *= kOut;
        if (whole) orow[e] = __float2bfloat16(sum > 0.f ? acc / sum : 0.f);
        else {
          part[e] = acc;
          if (d == 0) { part[a.group * 128 + head] = top; part[a.group * 129 + head] = sum; }
        }
      }
      if (!whole) {
        // the CTA that finishes the (row, kv head) last folds the partials of all (in CTA order: the same on every run)
        __threadfence();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (threadIdx.x == 0) *last_flag = atomicAdd(&sc.arrived[c.row * a.nkv + c.kvh], 1) == b1 - b0;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (*last_flag) {
          __threadfence();
          for (int e = threadIdx.x; e < a.group * 128; e += 256) {
            const int head = e >> 7;
            auto part_of = [&](int b) {
              const int start = static_cast<int>(static_cast<long long>(T) * b / G);
              return sc.partial + (static_cast<size_t>(b) * 2 + (start >= u0 ? 0 : (b == b0 ? 1 : 0))) * kDecPartial;
            };
            float top = -1e30f;
            for (int b = b0; b <= b1; ++b) top = fmaxf(top, __ldcg(part_of(b) + a.group * 128 + head));
            float acc = 0.f, sum = 0.f;
            for (int b = b0; b <= b1; ++b) {
              const float* q = part_of(b);
              const float f = dec_ex2(__ldcg(q + a.group * 128 + head) - top);
              acc += f * __ldcg(q + e);
              sum += f * __ldcg(q + a.group * 129 + head);
            }
            orow[e] = __float2bfloat16(sum > 0.f ? acc / sum : 0.f);
          }
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");        // the merge area is free again
    }
  }
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // give copies that were in flight when a role gave up time to land (bounded)
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) {}
  }
  __syncthreads();
}

}  // namespace plow
