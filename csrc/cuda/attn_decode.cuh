// Decode body of the grouped-query attention kernel: every row is one query token of its own sequence (head dim 128, at
// most 8 query heads per kv head), over the paged bf16 or e4m3 cache.
//
// A decode step reads each cached key and value once and does 2 x group multiply-adds per element, so it is bound by the
// stream from HBM.  The 128-lane tile form pays for its shape there: four heads fill 4 of 128 lanes, items of whole
// sequences leave SMs idle when lengths differ (170 us for 64 sequences of 512 to 4352 tokens, 98 us of traffic), and the
// e4m3 cache has to be rewritten as bf16 tiles in shared memory (268 us for half the traffic).  Here:
//   * all (row, kv head, page) triples of the step form one line, cut into equal pieces, one per CTA: every SM streams the
//     same number of pages.  A (row, kv head) that is cut leaves f32 partials; the CTA that finishes it last folds them.
//   * one warp feeds a ring of pages (TMA; the e4m3 scales by 4-byte cp.async), eight warps consume: two share a page, 32
//     tokens each, so four pages are in work at a time.  S = Q K^T (heads as rows) and O^T += V^T P^T (heads as columns) are
//     m16n8k16 warp MMAs: the accumulators of S are the B operand of the other one as they stand.  Every warp keeps its own
//     running maximum, sum and O, merged through shared memory by three other
//     warps when a piece ends (merged by the consumers themselves, CTAs with many short sequences took a third longer).
//   * e4m3 elements become f16 in registers, one conversion per pair (as bf16, by integer instructions, a pair took four and
//     the ALU pipe half the time); key scales multiply S, value scales P.  Q is scaled by a power of two into f16, which holds
//     every bf16 down to 2^-28 of the row's largest exactly; the running maximum is taken of score + log2(value scale), so
//     P times its value scale stays in f16's range.  There it has three more bits than in bf16 down to 2^-17 of the largest weight
//     of the warp, fewer below, and none below 2^-25: errors against 64 bits are the same or smaller up to 131072 tokens.  Cells that
//     no row sees may hold anything: their scores, value scales and value bytes are replaced on the pages that lo or hi cuts.  The
//     k index of an MMA may be any permutation as long as both operands agree, so a lane takes 16 consecutive bytes of a row.
// 64 sequences of 512 .. 4352 tokens, 32 / 8 heads, with the rotary writer: bf16 109 us (tile form 160 .. 169), e4m3 98 us
// (252 .. 263).  Both are near the stream rate: for 64 x 4096 tokens DRAM is 80 % (bf16) and 74 % busy.  Over the e4m3 cache 0.90 GB are
// read for 0.55 GB of cells, because a head's scale is 4 bytes of a 32-byte sector that the CTAs of eight heads fetch each for itself;
// issue slots are 40 % busy.
// The rates of mma.sync suffice by far (64 of 356 clocks per 16 tokens and SM).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "ptx.cuh"

namespace plow {

constexpr int kDecThreads = 384;          // 8 consumer warps, the producer warp, 3 merge warps
constexpr int kDecMaxCtas = 160;
constexpr int kDecMaxGroup = 8;
constexpr int kDecMaxRows = 256;
// Sequences of up to this many pages are not cut when each (row, kv head) can have a CTA of its own: 16 rows x 8 kv heads of 400
// tokens 16.5 us against 20.6 cut, of 800 tokens 18.5 / 22.6; 4 rows of 1000 tokens, e4m3, 20.6 / 18.5.
constexpr int kDecUncutPages = 12;
constexpr int kDecPartial = kDecMaxGroup * 130;      // floats of a partial: [head][128] O, then [head] m, [head] l

// Scratch of a call, in 4-byte words: plan (8), prefix of pages [rows + 1], arrivals [rows * nkv], partials [2 per CTA].
struct DecScratch {
  int* plan;            // [0]: 1 = this call is a decode step; [1]: pages; [2]: 1 = a CTA per (row, kv head)
  int* prefix;
  int* arrived;
  float* partial;
  __host__ __device__ DecScratch(void* base, int rows, int nkv) {
    plan = static_cast<int*>(base);
    prefix = plan + 8;
    arrived = prefix + rows + 1;
    // 16-byte vectors
    partial = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(arrived + rows * nkv) + 15) & ~static_cast<uintptr_t>(15));
  }
  static int64_t bytes(int rows, int nkv) {
    return 4ll * (8 + rows + 1 + static_cast<int64_t>(rows) * nkv + 2ll * kDecMaxCtas * kDecPartial) + 16;
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
  // A multiple of four: stage s then always belongs to the same two warps.  Otherwise a group would wait for some phases of a
  // stage only, and a parity wait cannot tell a phase from the one two before it.
  static constexpr int kStages = KV8 ? 8 : 4;
  static_assert(kStages % 4 == 0, "a stage belongs to one group of warps");
  // Pages whose scales are on their way.  The producer asks for a page once the one kStages before it is consumed, which it has then
  // long announced.
  static constexpr uint32_t kScaleLag = 3;
  static_assert(kScaleLag + 4 < kStages || !KV8, "every group of warps has a page that is announced");
  static constexpr int kTile = KV8 ? 8192 : 16384;               // one page of keys or values of a head
  static constexpr int kStage = 2 * kTile + (KV8 ? 512 : 0);     // + 64 key and 64 value scales
  // ring, control, then two merge areas: [8 warps][heads][132] f32
  static constexpr int kStageStride = (kStage + 1023) / 1024 * 1024;
  static constexpr int kRing = kStages * kStageStride;
  static constexpr int smem(int group) { return 1024 + kRing + 4096 + 2 * 8 * group * 132 * 4; }
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
__device__ __forceinline__ void mma_f16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two e4m3 bytes -> f16x2 (exact)
__device__ __forceinline__ uint32_t e4m3x2_to_f16(uint32_t x) {
  const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(x & 0xffffu), __NV_E4M3);
  return h.x | (static_cast<uint32_t>(h.y) << 16);
}
__device__ __forceinline__ uint32_t f16x2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float dec_ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
template <bool KV8>
__device__ void gqa_decode_body(const DecArgs& a, const CUtensorMap* tm_k, const CUtensorMap* tm_v) {
  using Cfg = DecCfg<KV8>;
  constexpr int kS = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* ctrl = ring + Cfg::kRing;
  uint64_t* full = reinterpret_cast<uint64_t*>(ctrl);        // [kS]
  uint64_t* empty = full + kS;                               // [kS]
  uint64_t* area_full = empty + kS;                          // [2]
  uint64_t* area_free = area_full + 2;                       // [2]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(area_free + 2);
  int* last_flag = const_cast<int*>(abort_flag) + 1;
  int* prefix = reinterpret_cast<int*>(ctrl + 512);          // [rows + 1]
  float* area = reinterpret_cast<float*>(ctrl + 4096);       // [2][8][group][132]: O, m, l
  const DecScratch sc(a.scratch, a.rows, a.nkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = sc.plan[1];
  const bool uncut = sc.plan[2] != 0;
  // pieces of at least four pages, which is what the warps have in work at a time
  const int G = uncut ? a.rows * a.nkv : min(static_cast<int>(gridDim.x), (T + 3) / 4);
  if (static_cast<int>(blockIdx.x) >= G) return;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kS; ++s) { mbar_init(&full[s], KV8 ? 2 : 1); mbar_init(&empty[s], 2); }
    for (int i = 0; i < 2; ++i) { mbar_init(&area_full[i], 8); mbar_init(&area_free[i], 3); }
    *abort_flag = 0;
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i <= a.rows; i += kDecThreads) prefix[i] = sc.prefix[i];
  __syncthreads();
  int p0 = static_cast<int>(static_cast<long long>(T) * blockIdx.x / G), p1 = static_cast<int>(static_cast<long long>(T) * (blockIdx.x + 1) / G);
  if (uncut) {
    const int row = blockIdx.x / a.nkv, n = (prefix[row + 1] - prefix[row]) / a.nkv;      // 0: an inactive row
    p0 = prefix[row] + (blockIdx.x % a.nkv) * n;
    p1 = p0 + n;
  }
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
            // scales of the 64 tokens: key scales, then value scales.  Lane 0 arrives for them once every lane has seen its own copies
            // of a page complete, kScaleLag pages later
            const float* src = a.kv_scale + static_cast<size_t>(page) * 64 * 2 * a.nkv + c.kvh;
            const uint32_t dst = smem_u32(st + 2 * Cfg::kTile);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int e = u * 32 + lane;
              const float* g = src + static_cast<size_t>(e & 63) * 2 * a.nkv + (e >= 64 ? a.nkv : 0);
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + e * 4), "l"(g) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (k >= Cfg::kScaleLag) {
              asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::kScaleLag) : "memory");
              __syncwarp();
              if (lane == 0) mbar_arrive(&full[(k - Cfg::kScaleLag) % kS]);
            }
          }
        }
      }
      p += c.n;
    }
    if constexpr (KV8) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      if (ok && lane == 0)
        for (uint32_t j = k > Cfg::kScaleLag ? k - Cfg::kScaleLag : 0; j < k; ++j) mbar_arrive(&full[j % kS]);
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ consumers
    const int group = warp >> 1, tok0 = (warp & 1) * 32;     // which of four pages in turn, which 32 of its tokens
    const int g = lane >> 2, c4 = lane & 3;
    uint32_t k0 = 0, n_piece = 0;                            // pages of the pieces before, pieces
    bool ok = true;
    for (int p = p0; ok && p < p1; ++n_piece) {
      const Piece c = piece_at(p);
      // Q fragments: MMA rows 0 .. 7 are the heads of this kv head, rows 8 .. 15 stay zero.  k-step s covers dims 16 s + {2 c4,
      // 2 c4 + 1, + 8, + 9}; for e4m3 dims 64 (s / 4) + 16 c4 + 4 (s % 4) + {0, 1, 2, 3} in the same places
      uint32_t qa[8][4];
      const __nv_bfloat16* qr = a.q + (static_cast<size_t>(c.row) * a.nq + c.kvh * a.group) * 128;
      float q_exp = 1.0f;                                    // e4m3: power of two that the scores are multiplied with again
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int d0 = KV8 ? 64 * (s >> 2) + 16 * c4 + 4 * (s & 3) : 16 * s + 2 * c4, d1 = KV8 ? d0 + 2 : d0 + 8;
        qa[s][0] = g < a.group ? *reinterpret_cast<const uint32_t*>(qr + g * 128 + d0) : 0u;
        qa[s][1] = 0u;
        qa[s][2] = g < a.group ? *reinterpret_cast<const uint32_t*>(qr + g * 128 + d1) : 0u;
        qa[s][3] = 0u;
      }
      if constexpr (KV8) {
        auto vals = [](uint32_t u) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u)); };
        float top = 0.f;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const float2 x = vals(qa[s][0]), y = vals(qa[s][2]);
          top = fmaxf(top, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(y.x), fabsf(y.y))));
        }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        // the exponent field of the largest moves to 2^14: scale = 2^(14 - e), its inverse goes into the scores
        const int e = min(max(static_cast<int>(__float_as_uint(top) >> 23) - 127, -100), 100);
        const float up = __uint_as_float(static_cast<uint32_t>(127 + 14 - e) << 23);
        q_exp = __uint_as_float(static_cast<uint32_t>(127 - 14 + e) << 23);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const float2 x = vals(qa[s][0]), y = vals(qa[s][2]);
          qa[s][0] = f16x2(x.x * up, x.y * up);
          qa[s][2] = f16x2(y.x * up, y.y * up);
        }
      }
      // O^T: m-tile n holds 16 dims (rows g, g + 8) by eight heads (columns 2 c4, 2 c4 + 1)
      float o[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[n][j] = 0.f;
      float m = -1e30f, l = 0.f;                             // of head g
      for (int i = (group - k0) & 3; ok && i < c.n; i += 4) {
        const uint32_t k = k0 + i;
        const int s = k % kS;
        if (!mbar_wait(&full[s], (k / kS) & 1, abort_flag)) { *abort_flag = 1; atomicCAS(a.status, 0, PLOW_ERR_TMA_WAIT | kTagGqa); ok = false; break; }
        const uint8_t* st = ring + s * Cfg::kStageStride;
        float sc4[4][4];                                     // S of tokens tok0 + 8 t + 2 c4 + {0, 1}, head g in [0], [1]
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int j = 0; j < 4; ++j) sc4[t][j] = 0.f;
        if constexpr (KV8) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const int row = tok0 + 8 * t + g;
              const uint4 w = *reinterpret_cast<const uint4*>(st + row * 128 + ((4 * h + c4) ^ (row & 7)) * 16);
              const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
              for (int u = 0; u < 4; ++u)
                mma_f16(sc4[t], qa[4 * h + u], e4m3x2_to_f16(ww[u]), e4m3x2_to_f16(ww[u] >> 16));
            }
        } else {
          // 8x8 blocks of an ldmatrix.x4: tokens 8 t .. + 7, dims 16 s .. + 15 and the next 16
          const uint32_t kb = smem_u32(st);
#pragma unroll
          for (int s2 = 0; s2 < 4; ++s2)
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const int row = tok0 + 8 * t + (lane & 7);
              const int chunk = 4 * s2 + (lane >> 3);        // 16-byte chunk of the 256-byte row
              uint32_t b[4];
              ldmatrix4(kb + (chunk >> 3) * 8192 + row * 128 + ((chunk & 7) ^ (row & 7)) * 16, b);
              mma_bf16(sc4[t], qa[2 * s2], b[0], b[1]);
              mma_bf16(sc4[t], qa[2 * s2 + 1], b[2], b[3]);
            }
        }
        float vs[8], lv[8];                                  // value scales and their log2
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int tok = tok0 + 8 * t + 2 * c4;
          float f0 = a.scale_log2e, f1 = a.scale_log2e;
          if constexpr (KV8) {
            const float* scs = reinterpret_cast<const float*>(st + 2 * Cfg::kTile);
            const float2 ks = *reinterpret_cast<const float2*>(scs + tok), v2 = *reinterpret_cast<const float2*>(scs + 64 + tok);
            const float f = a.scale_log2e * q_exp;
            f0 = ks.x * f; f1 = ks.y * f;
            vs[2 * t] = v2.x; vs[2 * t + 1] = v2.y;
            // a value scale of zero weighs nothing; the bound keeps exponentials over such tokens alone finite
            lv[2 * t] = fmaxf(__log2f(fabsf(v2.x)), -96.0f); lv[2 * t + 1] = fmaxf(__log2f(fabsf(v2.y)), -96.0f);
          }
          sc4[t][0] *= f0; sc4[t][1] *= f1;
        }
        const int t0 = (c.lo_page + c.first + i) * 64 + tok0;
        const bool edge = t0 < c.lo || t0 + 31 > c.hi;       // some of the 32 tokens are hidden
        if (edge) {
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int tok = t0 + 8 * t + 2 * c4 + j;
              if (tok < c.lo || tok > c.hi) {
                sc4[t][j] = -INFINITY;
                if constexpr (KV8) vs[2 * t + j] = 0.f;      // the cell may hold anything
              }
            }
        }
        // running maximum per head, moved only when exceeded by more than 2^7 (P then stays below that)
        float mx = -INFINITY;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if constexpr (KV8) mx = fmaxf(mx, fmaxf(sc4[t][0] + lv[2 * t], sc4[t][1] + lv[2 * t + 1]));
          else mx = fmaxf(mx, fmaxf(sc4[t][0], sc4[t][1]));
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const bool up = mx > m + 7.0f;
        if (__any_sync(0xffffffffu, up)) {
          const float n = up ? mx : m, f = dec_ex2(m - n);
          l *= f;
          m = n;
          const float f0 = __shfl_sync(0xffffffffu, f, 8 * c4), f1 = __shfl_sync(0xffffffffu, f, 8 * c4 + 4);    // heads 2 c4, 2 c4 + 1
#pragma unroll
          for (int j = 0; j < 8; ++j) { o[j][0] *= f0; o[j][1] *= f1; o[j][2] *= f0; o[j][3] *= f1; }
        }
        // P: the accumulator layout of S (head g, tokens 2 c4, 2 c4 + 1) is the B layout of the next MMA (column g, k 2 c4, ..)
        uint32_t pb[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          float e0 = dec_ex2(sc4[t][0] - m), e1 = dec_ex2(sc4[t][1] - m);
          l += e0 + e1;
          if constexpr (KV8) {
            pb[t] = f16x2(e0 * vs[2 * t], e1 * vs[2 * t + 1]);
          } else {
            const __nv_bfloat162 h0 = __floats2bfloat162_rn(e0, e1);
            pb[t] = *reinterpret_cast<const uint32_t*>(&h0);
          }
        }
        const uint8_t* vt = st + Cfg::kTile;
#pragma unroll
        for (int b16 = 0; b16 < 2; ++b16) {
          if constexpr (KV8) {
            // a lane takes 16 bytes (dims 16 g .. + 15) of the four tokens of its k indices; rows g and g + 8 of m-tile n are
            // dims 16 g + 2 n and 16 g + 2 n + 1
            uint32_t w[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int row = tok0 + 16 * b16 + 2 * c4 + (u & 1) + 8 * (u >> 1);
              const uint4 x = *reinterpret_cast<const uint4*>(vt + row * 128 + (g ^ (row & 7)) * 16);
              w[u][0] = x.x; w[u][1] = x.y; w[u][2] = x.z; w[u][3] = x.w;
            }
            if (edge) {                                      // NaN codes of hidden tokens would survive the weight zero
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int tok = t0 + 16 * b16 + 2 * c4 + (u & 1) + 8 * (u >> 1);
                if (tok < c.lo || tok > c.hi) w[u][0] = w[u][1] = w[u][2] = w[u][3] = 0u;
              }
            }
#pragma unroll
            for (int n = 0; n < 8; ++n) {
              // bytes 2 n, 2 n + 1 of tokens 2 c4 and 2 c4 + 1 (then + 8, + 9), side by side per dim
              const uint32_t sel = n & 1 ? 0x7362 : 0x5140;
              const uint32_t x = __byte_perm(w[0][n >> 1], w[1][n >> 1], sel), y = __byte_perm(w[2][n >> 1], w[3][n >> 1], sel);
              const uint32_t va[4] = {e4m3x2_to_f16(x), e4m3x2_to_f16(x >> 16), e4m3x2_to_f16(y), e4m3x2_to_f16(y >> 16)};
              mma_f16(o[n], va, pb[2 * b16], pb[2 * b16 + 1]);
            }
          } else {
            // 8x8 blocks: tokens 0 .. 7 of dims 16 n .. + 7 and + 8 .. + 15, then tokens 8 .. 15 of the same
            const uint32_t vb = smem_u32(vt);
            const int row = tok0 + 16 * b16 + (lane & 7) + 8 * (lane >> 4);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
              const int chunk = 2 * n + ((lane >> 3) & 1);
              uint32_t va[4];
              ldmatrix4_trans(vb + (chunk >> 3) * 8192 + row * 128 + ((chunk & 7) ^ (row & 7)) * 16, va);
              mma_bf16(o[n], va, pb[2 * b16], pb[2 * b16 + 1]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
      }
      k0 += c.n;
      p += c.n;
      // ---- the piece is done: this warp's partial (its tokens of the piece) to the merge warps
      const int buf = n_piece & 1;
      if (ok && !mbar_wait(&area_free[buf], ((n_piece >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; atomicCAS(a.status, 0, PLOW_ERR_STAGE_WAIT | kTagGqa); ok = false; }
      if (!ok) break;
      float* mine = area + (buf * 8 + warp) * a.group * 132;
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
      if (c4 == 0 && g < a.group) { mine[g * 132 + 128] = m; mine[g * 132 + 129] = l; }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int head = 2 * c4 + j;
        if (head < a.group) {
          float* dst = mine + head * 132;
#pragma unroll
          for (int n = 0; n < 8; ++n) {
            // dims of rows g and g + 8 of m-tile n
            dst[KV8 ? 16 * g + 2 * n : 16 * n + g] = o[n][j];
            dst[KV8 ? 16 * g + 2 * n + 1 : 16 * n + 8 + g] = o[n][2 + j];
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&area_full[buf]);
    }
  } else {
    // ------------------------------------------------------------------ merge warps
    // Every warp walks all pieces whatever its waits say (a wait that ran out is carried in `ok`), so the barriers of the
    // three cannot be left waiting.
    const int tid = threadIdx.x - 288;
    bool ok = true;
    uint32_t n_piece = 0;
    for (int p = p0; p < p1; ++n_piece) {
      const Piece c = piece_at(p);
      const bool is_first = p == p0;
      p += c.n;
      const int buf = n_piece & 1;
      if (ok && !mbar_wait(&area_full[buf], (n_piece >> 1) & 1, abort_flag)) { *abort_flag = 1; atomicCAS(a.status, 0, PLOW_ERR_TMEM_WAIT | kTagGqa); ok = false; }
      const int u0 = prefix[c.row] + c.kvh * c.pages;                              // the line's pages of this (row, kv head)
      const int b0 = static_cast<int>((static_cast<long long>(u0 + 1) * G - 1) / T), b1 = static_cast<int>((static_cast<long long>(u0 + c.pages) * G - 1) / T);
      const bool whole = uncut || b0 == b1;
      float* part = sc.partial + (static_cast<size_t>(blockIdx.x) * 2 + (is_first ? 0 : 1)) * kDecPartial;
      __nv_bfloat16* orow = a.out + (static_cast<size_t>(c.row) * a.nq + c.kvh * a.group) * 128;
      const int stride = a.group * 132;
      for (int e = tid * 4; ok && e < a.group * 128; e += 384) {                    // four dims of a head
        const int head = e >> 7, d = e & 127;
        const float* src = area + buf * 8 * stride + head * 132;
        float top = -1e30f, f[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) { f[w] = src[w * stride + 128]; top = fmaxf(top, f[w]); }
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          f[w] = dec_ex2(f[w] - top);
          const float4 x = *reinterpret_cast<const float4*>(src + w * stride + d);
          acc.x += f[w] * x.x; acc.y += f[w] * x.y; acc.z += f[w] * x.z; acc.w += f[w] * x.w;
          sum += f[w] * src[w * stride + 129];
        }
        if (whole) {
          const float inv = sum > 0.f ? 1.0f / sum : 0.f;
          const __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x * inv, acc.y * inv), hi = __floats2bfloat162_rn(acc.z * inv, acc.w * inv);
          *reinterpret_cast<uint2*>(orow + e) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
          *reinterpret_cast<float4*>(part + e) = acc;
          if (d == 0) { part[a.group * 128 + head] = top; part[a.group * 129 + head] = sum; }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&area_free[buf]);
      if (!whole) {
        // the CTA that finishes the (row, kv head) last folds the partials of all (in CTA order: the same on every run)
        __threadfence();
        asm volatile("bar.sync 1, 96;" ::: "memory");
        if (tid == 0) *last_flag = ok && atomicAdd(&sc.arrived[c.row * a.nkv + c.kvh], 1) == b1 - b0;
        asm volatile("bar.sync 1, 96;" ::: "memory");
        if (*last_flag) {
          __threadfence();
          // Eight partials' loads at a time (one by one, each waiting for L2, five to seven partials took 25 us).  Only the
          // first CTA may have started before this (row, kv head), which is then in its second place.
          const int first_place = static_cast<int>(static_cast<long long>(T) * b0 / G) >= u0 ? 0 : 1;
          for (int e = tid * 4; e < a.group * 128; e += 384) {
            const int head = e >> 7;
            float top = -1e30f, sum = 0.f;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int b = b0; b <= b1; b += 8) {
              float m[8], l[8];
              float4 x[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float* q = sc.partial + (static_cast<size_t>(b + j) * 2 + (b + j == b0 ? first_place : 0)) * kDecPartial;
                const bool in = b + j <= b1;
                m[j] = in ? __ldcg(q + a.group * 128 + head) : -1e30f;
                l[j] = in ? __ldcg(q + a.group * 129 + head) : 0.f;
                x[j] = in ? __ldcg(reinterpret_cast<const float4*>(q + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
              }
              float t = top;
#pragma unroll
              for (int j = 0; j < 8; ++j) t = fmaxf(t, m[j]);
              const float f0 = dec_ex2(top - t);
              top = t;
              acc.x *= f0; acc.y *= f0; acc.z *= f0; acc.w *= f0; sum *= f0;
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float f = dec_ex2(m[j] - t);
                acc.x += f * x[j].x; acc.y += f * x[j].y; acc.z += f * x[j].z; acc.w += f * x[j].w;
                sum += f * l[j];
              }
            }
            const float inv = sum > 0.f ? 1.0f / sum : 0.f;
            const __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x * inv, acc.y * inv), hi = __floats2bfloat162_rn(acc.z * inv, acc.w * inv);
            *reinterpret_cast<uint2*>(orow + e) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
          }
        }
        asm volatile("bar.sync 1, 96;" ::: "memory");       // the flag is read
      }
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
