// Flash attention for many query rows: grouped-query prefill (head dim 128) over the paged bf16 cache and materialised
// latent-attention prefill (192-wide keys, 128-wide values), on tcgen05.
//
// attn_gqa.cu serves every row count with one 128-lane tile per CTA: there the softmax of a tile and the MMAs of a tile
// take turns (tensor pipe 36 % busy, 523 TFLOP/s at 4096 tokens), and its 64-token key tiles make Q K^T read 6 KB of
// operands per 32 tensor clocks, more than shared memory delivers.  Here a CTA holds two query tiles, A and B, of the same
// kv head: eight warps of softmax per tile, and 128-token key tiles (two pages).  While the warps of one tile turn S into P
// the tensor core works for the other one:
//     ... P_A V (j), Q_A K^T (j+1), P_B V (j), Q_B K^T (j+1), P_A V (j+1) ...
// S (128 f32 columns; P, bf16, over the first 32 of each half) and O (128) of both tiles fill the 512 TMEM columns.  K and V come
// through one ring of 16 KB slabs (64 columns x 128 tokens) in the order they are used, so the ring holds 1.4 or 2 tiles
// for the two key widths.  The MMA warp runs straight on into the next item's first Q K^T, so an item's epilogue is hidden
// like any other softmax step.
//
// Items are (chunk of up to two tiles of consecutive rows, kv head); chunks are sorted by length on the device, items
// handed out through a counter, longest first, so the last ones are short.  With many heads they come in groups of as many
// heads as give every SM two items: the heads at work then share their keys in L2 (128 heads of 4096 tokens are 268 MB).  Masks, lazy rescaling
// and numerics are those of attn_gqa.cu.
//
// 4096 tokens, 32 / 8 heads: 154 to 158 us with the chunk list, the one-tile kernel with its list took 248 (890 to 868 against 554
// TFLOP/s); latent attention, 2048 rows behind 2048, 128 heads: 515 us against 632.  What bounds it: the chain of one tile
// (S ready, maximum, exponentials, P, P V, Q K^T, about 3000 clocks) is longer than the 2048 tensor clocks of the two tiles.
// Over a whole launch the tensor pipe is active 45 % (latent: 50 %) of the time, issue slots 46 %, the exponentials' pipe 36 %.  Tried and worse: an MMA warp per tile (166), waiting for the slabs
// before P instead of after (165).
#include <cuda_bf16.h>

#include "attn_prefill.h"
#include "ptx.cuh"
#include "tmap.cuh"

namespace plow {

namespace {

constexpr int kPage = 64;
constexpr int kThreads = 64 + 2 * 256;    // TMA, MMA, eight softmax warps for each of the two tiles
constexpr int kSlab = 128 * 128;          // 128 tokens x 64 bf16
constexpr int kItemRing = 4;
constexpr int kBuckets = 256;

// pad0, pad1: first and last row of a chunk while the list is made
struct Chunk { int r0, nt, page0, ntiles, last_page, slot, pad0, pad1; };

struct PfArgs {
  const int* page_table;
  const int* pos;
  const Chunk* chunks;
  const int* n_chunks;
  int* claim;
  __nv_bfloat16* out;
  int* status;
  int nq, nkv, group, max_pages, window;
  float scale_log2e;                      // > 0
  int negate;                             // the caller's scale is negative: scores change their sign first
  int kr;                                 // the last key slab comes from the shared rotary tensor
  int v_x0;                               // first value column within a head's row of the value tensor
};

template <int HDQ> struct PfCfg {
  static constexpr int kKS = HDQ / 64;                   // key slabs per tile
  static constexpr int kVS = 2;
  static constexpr int kSP = kKS + kVS;
  // K / V slabs in flight.  The next tile's K and V beside the V of this one are kSP + 2: fewer would deadlock.
  static constexpr int kRing = HDQ == 128 ? 8 : 7;
  static constexpr int kQTile = kKS * kSlab;
  static constexpr int kSmem = 1024 + 2 * kQTile + kRing * kSlab + 1024 + 4096;
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
  static_assert(kSP + kVS <= kRing, "the next tile beside this tile's values");
};

// One chunk per run of consecutive rows of a sequence, cut every `span` rows from the run's first one; sorted by length, longest
// first.  A span is two tiles, or one where the whole list then fits the chip at once (`sms` items or fewer; 256 rows behind
// 4000, 16 heads: 106 us with two, 89 with one).  One block: starts and ends are compacted separately in row order and pair up
// by index (kept in the last two words of the chunk slots), then a counting sort over quantised lengths fills the slots; the order
// within a bucket does not matter.  (Cuts at multiples of the span in the call's rows split runs shorter than a span: 100 runs of 15
// rows took 102 us, 94 now.)
__global__ void __launch_bounds__(1024)
prefill_chunks(const int* seq, const int* pos, int rows, int tq, int nkv, int sms, int window, Chunk* chunks, int cap, int* n_chunks, int* claim, int* status) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int count[kBuckets], first[kBuckets], cnt_s[32], cnt_e[32], last_s[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = threadIdx.x; b < kBuckets; b += blockDim.x) count[b] = 0;
  int n;
  for (int span = static_cast<long long>((rows + tq - 1) / tq) * nkv <= sms ? tq : 2 * tq;; span = 2 * tq) {
    n = 0;
    int n_e = 0, run0 = 0;                 // run0: first row of the run that the rows before r0 end with
    // position of row r, whether it goes on from the row before and to the row after
    struct Row { int p; bool from, on; };
    auto look = [&](int r) -> Row {
      const int p = r < rows ? pos[r] : -1, sq = r < rows ? seq[r] : 0;
      const int pb = r > 0 && r < rows ? pos[r - 1] : -1, pa = r + 1 < rows ? pos[r + 1] : -1;
      const int sb = r > 0 && r < rows ? seq[r - 1] : 0, sa = r + 1 < rows ? seq[r + 1] : 0;
      return Row{p, pb >= 0 && pb + 1 == p && sb == sq, pa >= 0 && p + 1 == pa && sa == sq};
    };
    Row next = look(threadIdx.x);
    for (int r0 = 0; r0 < rows; r0 += blockDim.x) {
      const int r = r0 + threadIdx.x, p = next.p;
      const bool from = next.from, on = next.on;
      next = look(r + blockDim.x);         // on its way during the barriers below
      const uint32_t fresh = __ballot_sync(0xffffffffu, !from), before = fresh & (0xffffffffu >> (31 - lane));
      if (lane == 0) last_s[warp] = fresh ? r + 31 - __clz(fresh) : -1;
      __syncthreads();
      const int ls = last_s[lane];
      const int r_warp = max(run0, __reduce_max_sync(0xffffffffu, lane < warp ? ls : -1));      // of the rows before this warp's
      const int r_run = before ? r - lane + 31 - __clz(before) : r_warp;
      run0 = max(run0, __reduce_max_sync(0xffffffffu, ls));
      const bool start = p >= 0 && (!from || (r - r_run) % span == 0), end = p >= 0 && (!on || (r + 1 - r_run) % span == 0);
      const uint32_t ms = __ballot_sync(0xffffffffu, start), me = __ballot_sync(0xffffffffu, end);
      if (lane == 0) { cnt_s[warp] = __popc(ms); cnt_e[warp] = __popc(me); }
      __syncthreads();
      const int vs = cnt_s[lane], ve = cnt_e[lane];
      const int at_s = n + __reduce_add_sync(0xffffffffu, lane < warp ? vs : 0) + __popc(ms & ((1u << lane) - 1));
      const int at_e = n_e + __reduce_add_sync(0xffffffffu, lane < warp ? ve : 0) + __popc(me & ((1u << lane) - 1));
      if (start && at_s < cap) chunks[at_s].pad0 = r;
      if (end && at_e < cap) chunks[at_e].pad1 = r;
      n += __reduce_add_sync(0xffffffffu, vs);
      n_e += __reduce_add_sync(0xffffffffu, ve);
    }
    if (span == 2 * tq || (n <= cap && static_cast<long long>(n) * nkv <= sms)) break;
    __syncthreads();
  }
  if (n > cap) {
    if (threadIdx.x == 0) atomicCAS(status, 0, PLOW_ERR_BOUNDS | kTagGqa);
    n = cap;
  }
  __syncthreads();
  auto chunk = [&](int i) -> Chunk {
    const int r = chunks[i].pad0, e = chunks[i].pad1;
    const int lo = window > 0 ? max(0, pos[r] - window + 1) : 0;
    Chunk c = {r, e - r + 1, lo / kPage, 0, pos[e] / kPage, seq[r], 0, 0};
    c.ntiles = (c.last_page - c.page0 + 2) / 2;
    return c;
  };
  auto bucket = [](int t) { return kBuckets - 1 - min(kBuckets - 1, t < 128 ? t : 96 + t / 4); };
  for (int i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&count[bucket(chunk(i).ntiles)], 1);
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int b0 = 0; b0 < kBuckets; b0 += 32) {
      const int v = count[b0 + lane];
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
      first[b0 + lane] = run + incl - v;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) { *n_chunks = n; *claim = 0; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const Chunk c = chunk(i);
    Chunk& o = chunks[atomicAdd(&first[bucket(c.ntiles)], 1)];
    o.r0 = c.r0; o.nt = c.nt; o.page0 = c.page0; o.ntiles = c.ntiles; o.last_page = c.last_page; o.slot = c.slot;
  }
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// 2^x of two values on the FMA pipe: x = n + f with n the nearest integer (the bits of x + 1.5 * 2^23 hold it), a degree-5
// minimax polynomial of 2^f on [-1/2, 1/2] (Remez fit; with its f32 roundings off by 2.1e-7 at most, 8e-8 rms, the same
// as ex2.approx), and n added to the exponent.  x <= 127; from -127 down (masked keys) the result is the smallest denormal, which is
// zero as a bf16.  A NaN comes out as the largest finite number, infinite as a bf16: a row's sum beyond kNanSum tells that it holds one
// (honest ones stay below 2^7 times the number of keys).
constexpr float kNanSum = 0x1p100f;
__device__ __forceinline__ float max_nan(float a, float b) { float r; asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void ex2_fma(float x0, float x1, float& r0, float& r1) {
  const f32x2 magic = pack2(12582912.0f, 12582912.0f), unmagic = pack2(-12582912.0f, -12582912.0f);
  const f32x2 x = pack2(max_nan(x0, -127.0f), max_nan(x1, -127.0f));
  const f32x2 t = add2(x, magic);
  const f32x2 f = fma2(add2(t, unmagic), pack2(-1.0f, -1.0f), x);
  f32x2 p = fma2(pack2(0.0013276472454890609f, 0.0013276472454890609f), f, pack2(0.009675540961325169f, 0.009675540961325169f));
  p = fma2(p, f, pack2(0.05550713092088699f, 0.05550713092088699f));
  p = fma2(p, f, pack2(0.24022120237350464f, 0.24022120237350464f));
  p = fma2(p, f, pack2(0.6931469440460205f, 0.6931469440460205f));
  p = fma2(p, f, pack2(1.0000001192092896f, 1.0000001192092896f));
  float t0, t1, p0, p1;
  unpack2(t, t0, t1);
  unpack2(p, p0, p1);
  r0 = __int_as_float(__float_as_int(p0) + (__float_as_int(t0) << 23));
  r1 = __int_as_float(__float_as_int(p1) + (__float_as_int(t1) << 23));
}

// What the roles of a CTA need of an item.
struct Work { int r0, nt, kvh, page0, ntiles, last_page, slot, pad; };

template <int HDQ>
__global__ void __launch_bounds__(kThreads, 1)
attn_prefill_kernel(const PfArgs a, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_kr) {
  pdl_launch_dependents();
  pdl_wait();
  using Cfg = PfCfg<HDQ>;
  constexpr int kKS = Cfg::kKS, kSP = Cfg::kSP, kRing = Cfg::kRing;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;                                // [2][kKS] slabs of 128 rows x 128 bytes
  uint8_t* ring = smem + 2 * Cfg::kQTile;
  uint8_t* ctrl = ring + kRing * kSlab;
  uint64_t* full = reinterpret_cast<uint64_t*>(ctrl);    // [kRing]
  uint64_t* empty = full + kRing;                        // [kRing]
  uint64_t* q_full = empty + kRing;
  uint64_t* q_empty = q_full + 1;
  uint64_t* s_full = q_empty + 1;                        // [2] by tile
  uint64_t* p_full = s_full + 2;                         // [2]
  uint64_t* p_half = p_full + 2;                         // [2] tokens 0 .. 63 of P are written (p_full: 64 .. 127)
  uint64_t* o_full = p_half + 2;                         // [2]
  uint64_t* o_free = o_full + 2;                         // [2]
  uint64_t* it_full = o_free + 2;                        // [kItemRing]
  uint64_t* it_empty = it_full + kItemRing;              // [kItemRing]
  uint64_t* drain_bar = it_empty + kItemRing;
  Work* items = reinterpret_cast<Work*>(drain_bar + 1);  // [kItemRing]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(items + kItemRing);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  volatile int* never_flag = abort_flag + 1;
  float* xch = reinterpret_cast<float*>(ctrl + 1024);    // [tile 2][parity 2][half 2][128 rows]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tq = 128 / a.group;                          // tokens per tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int g = 0; g < 2; ++g) { mbar_init(&s_full[g], 1); mbar_init(&p_full[g], 4); mbar_init(&p_half[g], 4); mbar_init(&o_full[g], 1); mbar_init(&o_free[g], 8); }
    for (int i = 0; i < kItemRing; ++i) { mbar_init(&it_full[i], 1); mbar_init(&it_empty[i], 17); }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    *never_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_kr);
  }
  if (warp == 1) { tmem_alloc(tmem_holder, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm_s = *tmem_holder;                    // S of tile g at + 128 g (P over 32 columns from 0 and from 64)
  const uint32_t tm_o = tm_s + 256;                      // O of tile g at + 128 g
  auto give_up = [&](int code) { *abort_flag = 1; atomicCAS(a.status, 0, code | kTagGqa); };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer; hands out the items
    if (elect_one()) {
      const int n_chunks = *a.n_chunks;
      const int n_items = n_chunks * a.nkv;
      const int head_group = a.nkv <= 16 ? a.nkv : max(1, min(a.nkv, 2 * static_cast<int>(gridDim.x) / max(1, n_chunks)));
      uint32_t slab = 0;
      bool ok = true;
      int n0 = 0, n1 = 0;                  // pages of the next tile to request
      // claims an item and posts it; its first pages are read at once, so that the loads wait for no dependent reads
      auto post = [&](uint32_t sq, Work& w) -> bool {
        const int idx = atomicAdd(a.claim, 1);
        w = Work{0, 0, 0, 0, 0, 0, 0, 0};
        if (idx < n_items) {
          // groups of heads, within a group by length
          const int grp = idx / (n_chunks * head_group), in = idx - grp * n_chunks * head_group;
          const int h0 = grp * head_group, nh = min(head_group, a.nkv - h0);
          const Chunk c = a.chunks[in / nh];
          w = Work{c.r0, c.nt, h0 + in % nh, c.page0, c.ntiles, c.last_page, c.slot, 0};
        }
        if (!mbar_wait(&it_empty[sq % kItemRing], ((sq / kItemRing) & 1) ^ 1, abort_flag)) { give_up(PLOW_ERR_STAGE_WAIT); return false; }
        items[sq % kItemRing] = w;
        mbar_arrive(&it_full[sq % kItemRing]);
        return true;
      };
      auto page_of = [&](const Work& w, int i) { return a.page_table[static_cast<size_t>(w.slot) * a.max_pages + min(i, w.last_page)]; };
      Work w, nx;
      ok = post(0, w);
      if (ok && w.nt > 0) { n0 = page_of(w, w.page0); n1 = page_of(w, w.page0 + 1); }
      for (uint32_t sq = 0; ok && w.nt > 0; ++sq, w = nx) {
        if (!mbar_wait(q_empty, (sq & 1) ^ 1, abort_flag)) { give_up(PLOW_ERR_STAGE_WAIT); break; }
        const int n_q = w.nt > tq ? 2 : 1;
        mbar_expect_tx(q_full, n_q * Cfg::kQTile);
        for (int g = 0; g < n_q; ++g)
          for (int c = 0; c < kKS; ++c) tma_load_3d(q_smem + g * Cfg::kQTile + c * kSlab, &tm_q, c * 64, w.kvh * a.group, w.r0 + g * tq, q_full);
        for (int j = 0; ok && j < w.ntiles; ++j) {
          const int p0 = n0 * kPage, p1 = n1 * kPage;
          if (j + 1 < w.ntiles) {
            n0 = page_of(w, w.page0 + 2 * j + 2);
            n1 = page_of(w, w.page0 + 2 * j + 3);       // past the end: the last page again, masked
          }
          for (int c = 0; c < kSP; ++c, ++slab) {
            const int s = slab % kRing;
            if (!mbar_wait(&empty[s], ((slab / kRing) & 1) ^ 1, abort_flag)) { give_up(PLOW_ERR_STAGE_WAIT); ok = false; break; }
            uint8_t* dst = ring + s * kSlab;
            mbar_expect_tx(&full[s], kSlab);
            const bool is_v = c >= kKS, is_r = a.kr && c == kKS - 1;
            const CUtensorMap* tm = is_v ? &tm_v : (is_r ? &tm_kr : &tm_k);
            const int x = is_v ? a.v_x0 + (c - kKS) * 64 : (is_r ? 0 : c * 64), y = is_r ? 0 : w.kvh;
            tma_load_3d(dst, tm, x, y, p0, &full[s]);
            tma_load_3d(dst + kSlab / 2, tm, x, y, p1, &full[s]);
          }
          if (ok && j == max(0, w.ntiles - 2)) ok = post(sq + 1, nx);      // late: an early claim would hold items back at the end
        }
        if (ok && nx.nt > 0) { n0 = page_of(nx, nx.page0); n1 = page_of(nx, nx.page0 + 1); }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc_qk = umma_idesc(128, 128, 1, 1);
      const uint32_t idesc_pv = umma_idesc(128, 128, 1, 1, 0, 1), idesc_pv_half = umma_idesc(128, 64, 1, 1, 0, 1);
      bool ok = true;
      auto get = [&](uint32_t sq, Work& w) -> bool {
        if (!mbar_wait(&it_full[sq % kItemRing], (sq / kItemRing) & 1, abort_flag)) { give_up(PLOW_ERR_TMA_WAIT); return false; }
        w = items[sq % kItemRing];
        mbar_arrive(&it_empty[sq % kItemRing]);
        return true;
      };
      auto slabs_here = [&](uint32_t first, int n) -> bool {
        for (int c = 0; c < n; ++c)
          if (!mbar_wait(&full[(first + c) % kRing], ((first + c) / kRing) & 1, abort_flag)) { give_up(PLOW_ERR_TMA_WAIT); return false; }
        tc_fence_after();
        return true;
      };
      auto release = [&](uint32_t first, int n) { for (int c = 0; c < n; ++c) tc_commit(&empty[(first + c) % kRing]); };
      // S_g = Q_g K^T of tile T.  S_g (and the P over it) was last read by P_g V of the tile before, issued earlier: the
      // tensor pipe executes in order.
      auto issue_qk = [&](int g, uint32_t T) -> bool {
        if (!slabs_here(T * kSP, kKS)) return false;
        const uint32_t qa = smem_u32(q_smem + g * Cfg::kQTile);
#pragma unroll
        for (int c = 0; c < kKS; ++c) {
          const uint64_t qd = umma_desc_k128(qa + c * kSlab), kd = umma_desc_k128(smem_u32(ring + ((T * kSP + c) % kRing) * kSlab));
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_f16(tm_s + g * 128, qd + 2 * k, kd + 2 * k, idesc_qk, (c | k) != 0);
        }
        tc_commit(&s_full[g]);
        return true;
      };
      // O_g += P_g V of tile T, in two halves of 64 tokens as P arrives
      auto issue_pv = [&](int g, uint32_t T, bool first, uint32_t parity) -> bool {
        if (!slabs_here(T * kSP + kKS, 2)) return false;
        const uint32_t v0 = (T * kSP + kKS) % kRing;
        const uint32_t va = smem_u32(ring + v0 * kSlab), vb = smem_u32(ring);
        const uint32_t p = tm_s + g * 128, o = tm_o + g * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!mbar_wait(h ? &p_full[g] : &p_half[g], parity, abort_flag)) { give_up(PLOW_ERR_TMEM_WAIT); return false; }
          tc_fence_after();
          if (v0 + 1 < kRing) {
#pragma unroll
            for (int j = 4 * h; j < 4 * h + 4; ++j)       // 16 tokens per MMA: two 8-token groups of 1024 bytes
              tc_mma_f16_ts(o, p + h * 32 + j * 8, umma_desc_mn128(va + j * 2048, kSlab, 1024), idesc_pv, !first || j != 0);
          } else {
            // the two value slabs lie at the two ends of the ring: one MMA per slab
#pragma unroll
            for (int j = 4 * h; j < 4 * h + 4; ++j) {
              tc_mma_f16_ts(o, p + h * 32 + j * 8, umma_desc_mn128(va + j * 2048, kSlab, 1024), idesc_pv_half, !first || j != 0);
              tc_mma_f16_ts(o + 64, p + h * 32 + j * 8, umma_desc_mn128(vb + j * 2048, kSlab, 1024), idesc_pv_half, !first || j != 0);
            }
          }
        }
        return true;
      };
      uint32_t sq = 0, Tq = 0, Tv = 0, n_p[2] = {0, 0}, n_it[2] = {0, 0};
      Work cur;
      ok = get(0, cur);
      bool more = ok && cur.nt > 0;
      if (more) {
        ok = mbar_wait(q_full, 0, abort_flag);
        if (!ok) give_up(PLOW_ERR_TMA_WAIT);
        tc_fence_after();
        ok = ok && issue_qk(0, Tq) && (cur.nt <= tq || issue_qk(1, Tq));
        if (ok) {
          release(Tq * kSP, kKS);
          ++Tq;
          if (cur.ntiles == 1) tc_commit(q_empty);
        }
      }
      int j = 0;
      while (ok && more) {
        const bool last = j + 1 == cur.ntiles, has_b = cur.nt > tq;
        Work nx = cur;
        if (last && !get(sq + 1, nx)) { ok = false; break; }
        const bool have_next = nx.nt > 0, nx_b = nx.nt > tq;
        for (int g = 0; g < 2; ++g) {
          if (g == 0 || has_b) {
            if (j == 0 && !mbar_wait(&o_free[g], (n_it[g] & 1) ^ 1, abort_flag)) { give_up(PLOW_ERR_TMEM_FREE_WAIT); ok = false; break; }
            if (!issue_pv(g, Tv, j == 0, n_p[g] & 1)) { ok = false; break; }
            ++n_p[g];
            if (last) { tc_commit(&o_full[g]); ++n_it[g]; }
          }
          if (g == (has_b ? 1 : 0)) release(Tv * kSP + kKS, 2);
          if (have_next && (g == 0 || nx_b)) {
            if (last && g == 0 && !mbar_wait(q_full, (sq + 1) & 1, abort_flag)) { give_up(PLOW_ERR_TMA_WAIT); ok = false; break; }
            tc_fence_after();
            if (!issue_qk(g, Tq)) { ok = false; break; }
          }
          if (have_next && g == (nx_b ? 1 : 0)) release(Tq * kSP, kKS);
        }
        if (!ok) break;
        ++Tv;
        more = have_next;
        if (!have_next) break;
        ++Tq;
        j = last ? 0 : j + 1;
        if (last) { cur = nx; ++sq; }
        if (j + 1 == cur.ntiles) tc_commit(q_empty);      // all Q K^T of the item are issued
      }
      if (!ok || *abort_flag) { tc_commit(drain_bar); mbar_wait(drain_bar, 0, never_flag); }
    }
  } else {
    // ------------------------------------------------------------------ softmax / epilogue warps of tile g
    // Two warps share a lane quarter, each with 64 of the 128 columns (and 64 of the accumulator's): one warp alone per
    // scheduler took 1350 clocks for its 128 exponentials, twice what the pipes need.
    const int g = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1;
    const int lq = warp & 3;             // TMEM lane quarter this warp may access
    const int li = lq * 32 + lane;       // row of the tile: token li / group, query head li % group
    const uint32_t lane_addr = static_cast<uint32_t>(lq * 32) << 16;
    const uint32_t ts = tm_s + g * 128 + lane_addr, to = tm_o + g * 128 + half * 64 + lane_addr;
    float* xg = xch + g * 512;
    uint32_t n_x = 0;
    // Both warps of a pair take the same way through everything below (their decisions come from values they share), so a
    // named barrier of the two cannot be left waiting; a wait that runs out is carried along in `live` until both leave.
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + g * 4 + lq) : "memory"); };
    // the other warp's value of this row; two buffers in turn, so one barrier per exchange is enough
    auto exchange = [&](float v) -> float {
      float* x = xg + (n_x & 1) * 256;
      ++n_x;
      x[half * 128 + li] = v;
      pair_sync();
      return x[(half ^ 1) * 128 + li];
    };
    const float c = a.scale_log2e;
    const f32x2 c2 = pack2(c, c);
    uint32_t n_s = 0, n_it = 0;
    bool live = true;
    for (uint32_t sq = 0;; ++sq) {
      if (live && !mbar_wait(&it_full[sq % kItemRing], (sq / kItemRing) & 1, abort_flag)) { give_up(PLOW_ERR_TMA_WAIT); live = false; }
      uint32_t stop;               // one decision for the pair
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, %2, 64, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                   : "=r"(stop) : "r"(static_cast<uint32_t>(!live)), "r"(1 + g * 4 + lq) : "memory");
      if (stop) break;
      const Work w = items[sq % kItemRing];
      __syncwarp();
      if (lane == 0) mbar_arrive(&it_empty[sq % kItemRing]);
      if (w.nt == 0) break;
      if (g == 1 && w.nt <= tq) continue;
      const int r0 = w.r0 + g * tq, nt = min(tq, w.nt - g * tq);
      const int n_valid = nt * a.group;
      const bool warp_active = lq * 32 < n_valid;         // whole warp: rows past the chunk are never read
      const int tok = min(li / a.group, nt - 1);
      const int hi = a.pos[r0 + tok];
      const int lo = a.window > 0 ? max(0, hi - a.window + 1) : 0;
      float m = -1e30f;
      f32x2 l0 = 0ull, l1 = 0ull;
      for (int j = 0; j < w.ntiles; ++j, ++n_s) {
        if (live && !mbar_wait(&s_full[g], n_s & 1, abort_flag)) { give_up(PLOW_ERR_TMEM_WAIT); live = false; }
        tc_fence_after();
        if (warp_active) {
          const int t0 = (w.page0 + 2 * j) * kPage + half * 64;
          const bool whole = __all_sync(0xffffffffu, t0 >= lo && t0 + 63 <= hi);
          uint32_t v[64];
          tmem_ld32(ts + half * 64, v);
          tmem_ld32(ts + half * 64 + 32, v + 32);
          tmem_ld_wait();
          if (a.negate) {
#pragma unroll
            for (int e = 0; e < 64; ++e) v[e] ^= 0x80000000u;
          }
          if (!whole) {
            const int rel_hi = hi - t0, rel_lo = lo - t0;
#pragma unroll
            for (int e = 0; e < 64; ++e) v[e] = e > rel_hi ? 0xff800000u : v[e];      // -inf
            if (a.window > 0) {
#pragma unroll
              for (int e = 0; e < 64; ++e) v[e] = e < rel_lo ? 0xff800000u : v[e];
            }
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int e = 0; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], __uint_as_float(v[e]));
          float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c;
          top = fmaxf(top, exchange(top));
          // lazy rescale: m only moves when a tile exceeds it by more than 2^kTau, so P <= 2^kTau and the accumulator in
          // TMEM is rarely touched.  P V of the tile before has retired: s_full was committed after it.
          constexpr float kTau = 7.0f;
          // +inf turns m, and with it the row's sum and accumulator, into NaN.
          const bool up = !(top <= m + kTau);
          if (__any_sync(0xffffffffu, up)) {               // the same in both warps of the pair
            const float m_new = up ? top + (top - top) : m;
            float s0, s1, s2, s3;
            unpack2(l0, s0, s1);
            unpack2(l1, s2, s3);
            const float alpha = fmaxf(fmaxf(s0, s1), fmaxf(s2, s3)) < kNanSum ? ex2(m - m_new) : NAN;
            const f32x2 al = pack2(alpha, alpha);
            l0 = fma2(l0, al, 0ull);
            l1 = fma2(l1, al, 0ull);
            m = m_new;
            if (j > 0) {
#pragma unroll 1
              for (int x = 0; x < 64; x += 16) {
                uint32_t o[16];
                tmem_ld16(to + x, o);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                tmem_st16(to + x, o);
              }
              tmem_st_wait();
              tc_fence_before();
              pair_sync();         // the first half of P V already adds to all columns
            }
          }
          const f32x2 nm = pack2(-m, -m);
          // P of a half lies over the first 32 of that half's own S columns, read already when they are written
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t pk[16];
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
              const uint32_t* u = v + q * 32 + e;
              const f32x2 x0 = fma2(pack2(__uint_as_float(u[0]), __uint_as_float(u[1])), c2, nm);
              const f32x2 x1 = fma2(pack2(__uint_as_float(u[2]), __uint_as_float(u[3])), c2, nm);
              float e0, e1, e2, e3;
              unpack2(x0, e0, e1);
              unpack2(x1, e2, e3);
              // 16 exponentials a clock and SM against 4096 MACs: for 128-wide heads ex2 alone takes as long as both MMAs.
              // A quarter of them goes to the FMA pipe (4096 tokens: a quarter 152 us, three eighths 154, half 158).
              const int pair = (e >> 1) & 7;
              if (pair == 4) ex2_fma(e0, e1, e0, e1); else { e0 = ex2(e0); e1 = ex2(e1); }
              if (pair == 0) ex2_fma(e2, e3, e2, e3); else { e2 = ex2(e2); e3 = ex2(e3); }
              l0 = add2(l0, pack2(e0, e1));
              l1 = add2(l1, pack2(e2, e3));
              const __nv_bfloat162 h0 = __floats2bfloat162_rn(e0, e1), h1 = __floats2bfloat162_rn(e2, e3);
              pk[e >> 1] = *reinterpret_cast<const uint32_t*>(&h0);
              pk[(e >> 1) + 1] = *reinterpret_cast<const uint32_t*>(&h1);
            }
            tmem_st16(ts + half * 64 + q * 16, pk);
          }
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(half ? &p_full[g] : &p_half[g]);
      }
      if (live && !mbar_wait(&o_full[g], n_it & 1, abort_flag)) { give_up(PLOW_ERR_TMEM_WAIT); live = false; }
      ++n_it;
      tc_fence_after();
      if (warp_active) {
        float s0, s1, s2, s3;
        unpack2(l0, s0, s1);
        unpack2(l1, s2, s3);
        const float l_own = (s0 + s1) + (s2 + s3), l_other = exchange(l_own);
        const float l = l_own + l_other;
        const float fin = l > 0.f ? (l < kNanSum ? 1.0f / l : NAN) : 0.f;      // a NaN sum: the accumulator holds them too
        const bool row_ok = li < n_valid;
        uint4* dst = reinterpret_cast<uint4*>(a.out + (static_cast<size_t>(r0 + li / a.group) * a.nq + w.kvh * a.group + li % a.group) * 128 + half * 64);
#pragma unroll 1
        for (int x = 0; x < 64; x += 32) {
          uint32_t o[32];
          __syncwarp();
          tmem_ld32(to + x, o);
          tmem_ld_wait();
          if (!row_ok || !live) continue;
          uint32_t h2[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(o[2 * e]) * fin, __uint_as_float(o[2 * e + 1]) * fin);
            h2[e] = *reinterpret_cast<const uint32_t*>(&v);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) dst[x / 8 + q] = make_uint4(h2[4 * q], h2[4 * q + 1], h2[4 * q + 2], h2[4 * q + 3]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_free[g]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // give TMA copies that were in flight when a role gave up time to land (bounded)
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) {}
  }
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tm_s, 512); }
}

template <int HDQ>
int launch(const PrefillArgs& p, const PfArgs& a, cudaStream_t stream) {
  using Cfg = PfCfg<HDQ>;
  CUtensorMap tq, tk, tv, tr;
  const uint64_t n = static_cast<uint64_t>(p.n_tokens);
  int r = make_tmap_3d(&tq, p.q, 2, HDQ, p.nq, p.rows, HDQ * 2, static_cast<uint64_t>(p.nq) * HDQ * 2, a.group, 128 / a.group, 128);
  if (r) return 1100 + r;
  if (p.kr) {
    r = make_tmap_3d(&tk, p.k, 2, 256, p.nkv, n, 256 * 2, static_cast<uint64_t>(p.nkv) * 256 * 2, 1, kPage, 128);
    if (r) return 1200 + r;
    tv = tk;
    r = make_tmap_3d(&tr, p.kr, 2, 64, 1, n, 64 * 2, 64 * 2, 1, kPage, 128);
    if (r) return 1300 + r;
  } else {
    r = make_tmap_3d(&tk, p.k, 2, HDQ, p.nkv, n, HDQ * 2, static_cast<uint64_t>(p.nkv) * HDQ * 2, 1, kPage, 128);
    if (r) return 1200 + r;
    r = make_tmap_3d(&tv, p.v, 2, 128, p.nkv, n, 128 * 2, static_cast<uint64_t>(p.nkv) * 128 * 2, 1, kPage, 128);
    if (r) return 1300 + r;
    tr = tk;
  }
  static DeviceOnce attr;
  if (ensure_smem(attr, attn_prefill_kernel<HDQ>, Cfg::kSmem) != cudaSuccess) return 3000;
  launch_serial(attn_prefill_kernel<HDQ>, dim3(sm_count()), dim3(kThreads), Cfg::kSmem, stream, a, tq, tk, tv, tr);
  return 0;
}

}  // namespace

int launch_attn_prefill(const PrefillArgs& p, cudaStream_t stream) {
  PfArgs a;
  a.page_table = p.page_table; a.pos = p.pos; a.chunks = static_cast<const Chunk*>(p.chunks); a.n_chunks = p.counters; a.claim = p.claim;
  a.out = static_cast<__nv_bfloat16*>(p.out); a.status = p.status;
  a.nq = p.nq; a.nkv = p.nkv; a.group = p.nq / p.nkv; a.max_pages = p.max_pages; a.window = p.window;
  // masked scores are -inf before the scale: it stays positive and non-zero
  a.negate = p.scale < 0.f ? 1 : 0;
  a.scale_log2e = fmaxf(fabsf(p.scale) * 1.4426950408889634f, 1e-30f);
  a.kr = p.kr ? 1 : 0; a.v_x0 = p.kr ? 128 : 0;
  launch_serial(prefill_chunks, dim3(1), dim3(1024), 0, stream, p.seq, p.pos, p.rows, 128 / a.group, p.nkv, sm_count(), p.window,
                static_cast<Chunk*>(p.chunks), p.chunk_cap, p.counters, p.claim, p.status);
  return p.kr ? launch<192>(p, a, stream) : launch<128>(p, a, stream);
}

}  // namespace plow

