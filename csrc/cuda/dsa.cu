// Sparse-attention "lightning indexer": index-key cache write, index scores on tcgen05, exact top-k.
//
//   k_idx[t]   = RoPE(LayerNorm(wk x_t) * gamma + beta)                    -> e4m3 row + f32 scale, paged
//   score[r,t] = sum_h w[r,h] * ReLU(q_idx[r,h] . k_idx[t])                 for t <= pos[r]
//   sel[r]     = the top_k positions by (score desc, lowest index on ties);  rows with at most top_k
//                visible positions emit the identity, trailing slots are -1.
// Reference semantics: runtime/common/dev_isa.h:516-534 and :1083-1115 (7-pass radix select over a
// monotone packed key, live token-granular kv_len), runtime/nvidia/op_dsa.cuh.
//
// Scores: one CTA per (up to eight 128-token tiles, query row).  A tile's keys are the A operand (M = 128 tokens),
// the row's 64 index heads the B operand (N = 64), K = 128 e4m3: D[token][head] lands with one token
// per TMEM lane, so the weighted ReLU sum over heads is a private 64-column loop per thread and the
// score leaves the kernel with one coalesced store.  One warp keeps a ring of four tiles and two accumulators busy,
// four warps read them back; three CTAs per SM.  DRAM is half busy while it runs; the warps wait for the keys' scales and
// the read-back.  (A CTA per tile paid
// barrier and TMEM set-up and one exposed TMA -> MMA -> read-back chain for every 16 KB: 106 us for 64 rows x 32768,
// 68 us now.)
//
// Top-k: one cluster per row, the row's scores in shared memory as monotone integer keys.  A counting pass over 2048 bins
// of the key range finds the bin that holds the cut; its elements (a few hundred) are sorted by the first CTA, which gives
// the cut value and how many of its ties are taken, lowest index first; a last pass writes the selection in index order.
// (One CTA per row took seven 8-bit digit passes over
// global memory: 121 us for 64 rows x 32768, top 2048; 51 to 65 us now, half of the stalls at the barriers of CTAs and clusters.)
#include <cuda_bf16.h>
#include <cooperative_groups.h>
#include <cuda_fp8.h>

#include "ptx.cuh"
#include "tmap.cuh"

namespace plow {

constexpr int kIdxDim = 128;
constexpr int kIdxHeads = 64;
constexpr int kIdxPage = 64;

// One warp per row: LayerNorm (+bias), RoPE on the first `rot` dims, e4m3 quantisation with one scale.
__global__ void dsa_k_write_kernel(uint8_t* cache, float* cache_scale, const __nv_bfloat16* k, int ld_k,
                                   const float* gamma, const float* beta, const float* rope_tab, const int* pos,
                                   const int* seq, const int* page_table, int max_pages, int rows, int rot,
                                   int pair_mode, float eps) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  __shared__ float buf[8][kIdxDim];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * 8 + wib;
  if (r >= rows) return;
  const int p = pos[r];
  if (p < 0) return;
  float v[4], s = 0.f, ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[j] = __bfloat162float(k[static_cast<size_t>(r) * ld_k + lane + 32 * j]); s += v[j]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float mean = s / kIdxDim;
#pragma unroll
  for (int j = 0; j < 4; ++j) { v[j] -= mean; ss += v[j] * v[j]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rs = rsqrtf(ss / kIdxDim + eps);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = lane + 32 * j;
    buf[wib][c] = v[j] * rs * gamma[c] + (beta ? beta[c] : 0.f);
  }
  __syncwarp();
  const int half = rot / 2;
  const float* tab = rope_tab + static_cast<size_t>(p) * rot;
  float o4[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = lane + 32 * j;
    float y = buf[wib][c];
    if (c < rot) {
      int i, partner; bool first;
      if (pair_mode) { i = c >> 1; first = !(c & 1); partner = c ^ 1; }
      else { first = c < half; i = first ? c : c - half; partner = first ? c + half : c - half; }
      const float x = buf[wib][c], z = buf[wib][partner], cs = tab[i], sn = tab[half + i];
      y = first ? x * cs - z * sn : x * cs + z * sn;
    }
    o4[j] = y;
  }
  float amax = fmaxf(fmaxf(fabsf(o4[0]), fabsf(o4[1])), fmaxf(fabsf(o4[2]), fabsf(o4[3])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float sc = fmaxf(amax, 1e-10f) / 448.0f, inv = 1.0f / sc;
  const int page = page_table[static_cast<size_t>(seq[r]) * max_pages + p / kIdxPage];
  const size_t cell = static_cast<size_t>(page) * kIdxPage + p % kIdxPage;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_fp8_e4m3 q(o4[j] * inv);
    cache[cell * kIdxDim + lane + 32 * j] = *reinterpret_cast<const uint8_t*>(&q);
  }
  if (lane == 0) cache_scale[cell] = sc;
}

// One warp per (row, head): RoPE on the first `rot` dims, e4m3 with one scale; the scale and the head
// weight are folded into w_out[r][h] = w[r][h] * scale so the score kernel multiplies once.
__global__ void dsa_q_prep_kernel(uint8_t* q8, float* w_out, const __nv_bfloat16* q, int ld_q, const float* w, int ld_w,
                                  const float* rope_tab, const int* pos, int rows, int rot, int pair_mode) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  __shared__ float buf[8][kIdxDim];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * 8 + wib;
  if (item >= rows * kIdxHeads) return;
  const int r = item / kIdxHeads, h = item % kIdxHeads;
  const int p = max(pos[r], 0);
#pragma unroll
  for (int j = 0; j < 4; ++j) buf[wib][lane + 32 * j] = __bfloat162float(q[static_cast<size_t>(r) * ld_q + h * kIdxDim + lane + 32 * j]);
  __syncwarp();
  const int half = rot / 2;
  const float* tab = rope_tab + static_cast<size_t>(p) * rot;
  float o4[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = lane + 32 * j;
    float y = buf[wib][c];
    if (c < rot) {
      int i, partner; bool first;
      if (pair_mode) { i = c >> 1; first = !(c & 1); partner = c ^ 1; }
      else { first = c < half; i = first ? c : c - half; partner = first ? c + half : c - half; }
      const float x = buf[wib][c], z = buf[wib][partner], cs = tab[i], sn = tab[half + i];
      y = first ? x * cs - z * sn : x * cs + z * sn;
    }
    o4[j] = y;
  }
  float amax = fmaxf(fmaxf(fabsf(o4[0]), fabsf(o4[1])), fmaxf(fabsf(o4[2]), fabsf(o4[3])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float sc = fmaxf(amax, 1e-10f) / 448.0f, inv = 1.0f / sc;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_fp8_e4m3 e(o4[j] * inv);
    q8[(static_cast<size_t>(r) * kIdxHeads + h) * kIdxDim + lane + 32 * j] = *reinterpret_cast<const uint8_t*>(&e);
  }
  if (lane == 0) w_out[r * kIdxHeads + h] = w[static_cast<size_t>(r) * ld_w + h] * sc;
}

constexpr int kScoreTiles = 8;            // 128-token tiles per CTA at most
constexpr int kScoreStages = 4;
constexpr int kScoreSmem = 1024 + 8192 + kScoreStages * 16384 + 1024;

__global__ void __launch_bounds__(160)
dsa_score_kernel(float* scores, int ld_scores, int cta_tiles, const float* w, const float* kscale, const int* pos, const int* seq,
                 const int* page_table, int max_pages, int* status, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_q) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const int r = blockIdx.y, t0 = blockIdx.x * 128 * cta_tiles;
  const int len = pos[r] + 1;
  if (t0 >= len) return;
  const int n_tiles = min(cta_tiles, (len - t0 + 127) / 128);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;                 // 64 heads x 128 B
  uint8_t* k_smem = smem + 8192;          // [stage] 128 tokens x 128 B
  uint64_t* full = reinterpret_cast<uint64_t*>(k_smem + kScoreStages * 16384);     // [stage]
  uint64_t* empty = full + kScoreStages;                                           // [stage]
  uint64_t* acc_full = empty + kScoreStages;                                       // [2]
  uint64_t* acc_empty = acc_full + 2;                                              // [2]
  uint64_t* drain_bar = acc_empty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  volatile int* never_flag = abort_flag + 1;
  float* w_smem = reinterpret_cast<float*>(full) + 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kScoreStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    *never_flag = 0;
    fence_mbar_init();
  }
  if (threadIdx.x < kIdxHeads) w_smem[threadIdx.x] = w[r * kIdxHeads + threadIdx.x];
  if (warp == 4) { tmem_alloc(tmem_holder, 128); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tmem_holder;
  const int* pt = page_table + static_cast<size_t>(seq[r]) * max_pages + t0 / kIdxPage;
  const int last_page = (len - 1 - t0) / kIdxPage;
  if (warp == 4) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc(128, 64, 0, 0);
      bool ok = true;
      auto load = [&](int i) -> bool {
        const int s = i % kScoreStages;
        if (!mbar_wait(&empty[s], ((i / kScoreStages) & 1) ^ 1, abort_flag)) { *abort_flag = 1; atomicCAS(status, 0, PLOW_ERR_STAGE_WAIT | kTagDsa); return false; }
        // the second half of the last tile may lie past the row: its last page again, never stored
        mbar_expect_tx(&full[s], 16384 + (i == 0 ? 8192 : 0));
        tma_load_2d(k_smem + s * 16384, &tm_k, 0, pt[2 * i] * kIdxPage, &full[s]);
        tma_load_2d(k_smem + s * 16384 + 8192, &tm_k, 0, pt[min(2 * i + 1, last_page)] * kIdxPage, &full[s]);
        if (i == 0) tma_load_2d(q_smem, &tm_q, 0, r * kIdxHeads, &full[s]);
        return true;
      };
      for (int i = 0; ok && i < min(kScoreStages, n_tiles); ++i) ok = load(i);
      const uint64_t qd = umma_desc_k128(smem_u32(q_smem));
      for (int i = 0; ok && i < n_tiles; ++i) {
        const int s = i % kScoreStages, b = i & 1;
        if (!mbar_wait(&acc_empty[b], ((i >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; atomicCAS(status, 0, PLOW_ERR_TMEM_FREE_WAIT | kTagDsa); ok = false; break; }
        if (!mbar_wait(&full[s], (i / kScoreStages) & 1, abort_flag)) { *abort_flag = 1; atomicCAS(status, 0, PLOW_ERR_TMA_WAIT | kTagDsa); ok = false; break; }
        tc_fence_after();
        const uint64_t kd = umma_desc_k128(smem_u32(k_smem + s * 16384));
#pragma unroll
        for (int k = 0; k < 4; ++k) tc_mma_f8(tm + b * 64, kd + 2 * k, qd + 2 * k, idesc, k > 0);
        tc_commit(&empty[s]);
        tc_commit(&acc_full[b]);
        if (i + kScoreStages < n_tiles) ok = load(i + kScoreStages);
      }
      if (!ok) { tc_commit(drain_bar); mbar_wait(drain_bar, 0, never_flag); }
    }
    __syncwarp();
  } else {
    const uint32_t lane_addr = static_cast<uint32_t>(warp * 32) << 16;
    for (int i = 0; i < n_tiles; ++i) {
      const int b = i & 1, t = t0 + i * 128 + static_cast<int>(threadIdx.x);
      // the key's scale is on its way while the MMAs run
      float ks = 0.f;
      if (t < len) ks = kscale[static_cast<size_t>(pt[2 * i + (threadIdx.x >> 6)]) * kIdxPage + (t % kIdxPage)];
      if (!mbar_wait(&acc_full[b], (i >> 1) & 1, abort_flag)) { *abort_flag = 1; atomicCAS(status, 0, PLOW_ERR_TMEM_WAIT | kTagDsa); break; }
      tc_fence_after();
      uint32_t d[64];
      tmem_ld32(tm + b * 64 + lane_addr, d);
      tmem_ld32(tm + b * 64 + lane_addr + 32, d + 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[b]);
      float acc = 0.f;
#pragma unroll
      for (int h = 0; h < 64; ++h) acc = fmaf(w_smem[h], fmaxf(__uint_as_float(d[h]), 0.f), acc);
      if (t < len) scores[static_cast<size_t>(r) * ld_scores + t] = acc * ks;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // give copies that were in flight when a role gave up time to land (bounded)
    const unsigned long long c0 = globaltimer_ns();
    while (globaltimer_ns() - c0 < 2000000ull) {}
  }
  __syncthreads();
  if (warp == 4) { tc_fence_after(); tmem_dealloc(tm, 128); }
}

constexpr int kTopThreads = 512;
constexpr int kTopWarps = kTopThreads / 32;
constexpr int kTopBins = 2048;
constexpr int kTopCap = 2048;             // elements of the bin that holds the cut; more: the bin is cut into bins again
constexpr int kTopCluster = 8;
constexpr int kTopSlice = 40960;          // keys of a row a CTA keeps in shared memory; longer rows are read again

__device__ __forceinline__ uint32_t dsa_key(float s) {      // monotone, NaN above everything (by its bits)
  const uint32_t b = __float_as_uint(s);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct TopShared {
  uint32_t part[2][4];                    // this CTA's share of a cluster-wide result; two buffers in turn
  uint32_t bcast[4];
  uint32_t red[kTopWarps], red2[kTopWarps];
  int list_n;
};

__global__ void __launch_bounds__(kTopThreads)
dsa_topk_kernel(int* sel, const float* scores, int ld_scores, const int* pos, int top_k, int slice_cap) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) uint32_t top_smem[];
  uint32_t* hist = top_smem;              // [kTopBins]
  uint32_t* list = hist + kTopBins;       // [kTopCap] the first CTA's: keys of the cut's bin
  uint32_t* keys = list + kTopCap;        // [slice_cap]
  __shared__ TopShared sh;
  const int nc = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
  const int row = blockIdx.x / nc;
  const int len = pos[row] + 1;
  int* out = sel + static_cast<size_t>(row) * top_k;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (len <= top_k) {                     // the same for the whole cluster
    for (int j = rank * kTopThreads + tid; j < top_k; j += nc * kTopThreads) out[j] = j < len ? j : -1;
    return;
  }
  const int slice = ((len + nc - 1) / nc + 31) & ~31;
  const int base = min(len, rank * slice), n = min(len, base + slice) - base;
  const float* src = scores + static_cast<size_t>(row) * ld_scores + base;
  const bool in_smem = slice <= slice_cap;
  auto key_at = [&](int i) { return in_smem ? keys[i] : dsa_key(src[i]); };
  // smallest and largest key
  uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll 8
  for (int i = tid; i < n; i += kTopThreads) {
    const uint32_t k = dsa_key(src[i]);
    if (in_smem) keys[i] = k;
    lo = min(lo, k); hi = max(hi, k);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) { sh.red[warp] = lo; sh.red2[warp] = hi; }
  __syncthreads();
  int ex = 0;
  if (warp == 0) {
    lo = __reduce_min_sync(0xffffffffu, lane < kTopWarps ? sh.red[lane] : 0xFFFFFFFFu);
    hi = __reduce_max_sync(0xffffffffu, lane < kTopWarps ? sh.red2[lane] : 0u);
    if (lane == 0) { sh.part[ex][0] = lo; sh.part[ex][1] = hi; }
  }
  cl.sync();
  lo = 0xFFFFFFFFu; hi = 0;
  for (int q = 0; q < nc; ++q) {
    const TopShared* o = cl.map_shared_rank(&sh, q);
    lo = min(lo, o->part[ex][0]); hi = max(hi, o->part[ex][1]);
  }
  ex ^= 1;
  uint32_t above = 0;                     // elements with keys over `hi`: taken in any case
  uint32_t own = 0;                       // elements in [lo, hi], which holds the cut
  while (true) {
    // (hi - lo) >> shift < kTopBins; bin 0 holds the largest keys
    const int shift = max(0, 21 - __clz(hi - lo));
    for (int i = tid; i < kTopBins; i += kTopThreads) hist[i] = 0;
    if (tid == 0) sh.list_n = 0;
    __syncthreads();
    for (int i = tid; i < n; i += kTopThreads) {
      const uint32_t k = key_at(i);
      if (k >= lo && k <= hi) atomicAdd(&hist[(hi - k) >> shift], 1u);
    }
    cl.sync();
    // every CTA sums the same histogram: four neighbouring bins per thread, then a prefix over the threads
    uint4 h = make_uint4(0u, 0u, 0u, 0u);
    for (int q = 0; q < nc; ++q) {
      const uint4 v = reinterpret_cast<const uint4*>(cl.map_shared_rank(hist, q))[tid];
      h.x += v.x; h.y += v.y; h.z += v.z; h.w += v.w;
    }
    const uint32_t mine = h.x + h.y + h.z + h.w;
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
    if (lane == 31) sh.red[warp] = incl;
    __syncthreads();
    uint32_t before = above + incl - mine;
    for (int w = 0; w < warp; ++w) before += sh.red[w];
    // the one thread whose bins reach top_k names the bin
    const uint32_t want = static_cast<uint32_t>(top_k);
    if (before < want && before + mine >= want) {
      const uint32_t hv[4] = {h.x, h.y, h.z, h.w};
      uint32_t acc = before;
      int b = 0;
      while (acc + hv[b] < want) acc += hv[b++];
      sh.bcast[0] = 4 * tid + b; sh.bcast[1] = acc; sh.bcast[2] = hv[b];
    }
    __syncthreads();
    const uint32_t bin = sh.bcast[0];
    above = sh.bcast[1]; own = sh.bcast[2];
    const uint32_t new_hi = hi - (bin << shift), w = (1u << shift) - 1;
    lo = new_hi - lo > w ? new_hi - w : lo;
    hi = new_hi;
    cl.sync();                            // all have read the histograms
    if (own <= kTopCap || lo == hi) break;
  }
  uint32_t cut = lo, ties;                // keys over `cut` are taken, and the first `ties` that equal it
  if (lo == hi) {
    ties = top_k - above;
  } else {
    // the bin's keys to the first CTA
    uint32_t* l0 = cl.map_shared_rank(list, 0);
    int* n0 = &cl.map_shared_rank(&sh, 0)->list_n;
    for (int i = tid; i < n; i += kTopThreads) {
      const uint32_t k = key_at(i);
      if (k >= lo && k <= hi) l0[atomicAdd(n0, 1)] = k;
    }
    cl.sync();
    if (rank == 0) {
      int n2 = 32;
      while (n2 < static_cast<int>(own)) n2 <<= 1;
      for (int i = static_cast<int>(own) + tid; i < n2; i += kTopThreads) list[i] = 0;
      for (int size = 2; size <= n2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          __syncthreads();
          for (int t = tid; t < n2 / 2; t += kTopThreads) {
            const int i = 2 * t - (t & (stride - 1)), j = i + stride;
            const uint32_t x = list[i], y = list[j];
            if ((x < y) == ((i & size) == 0)) { list[i] = y; list[j] = x; }
          }
        }
      __syncthreads();
      const int need = top_k - static_cast<int>(above);       // of the sorted list
      const uint32_t c = list[need - 1];
      int larger = 0;
      for (int i = tid; i < need; i += kTopThreads) larger += list[i] > c;
      larger = __reduce_add_sync(0xffffffffu, larger);
      if (lane == 0) sh.red[warp] = larger;
      __syncthreads();
      if (tid == 0) {
        int total = 0;
        for (int q = 0; q < kTopWarps; ++q) total += sh.red[q];
        sh.bcast[0] = c; sh.bcast[1] = need - total;
      }
    }
    cl.sync();
    cut = cl.map_shared_rank(&sh, 0)->bcast[0];
    ties = cl.map_shared_rank(&sh, 0)->bcast[1];
  }
  // counts of larger and equal keys before this warp's part, then the selection in index order
  const int seg = ((n + kTopWarps - 1) / kTopWarps + 31) & ~31;
  const int s0 = min(n, warp * seg), s1 = min(n, s0 + seg);
  int gt = 0, eq = 0;
  for (int i = s0 + lane; i < s1; i += 32) { const uint32_t k = key_at(i); gt += k > cut; eq += k == cut; }
  gt = __reduce_add_sync(0xffffffffu, gt);
  eq = __reduce_add_sync(0xffffffffu, eq);
  __syncthreads();
  if (lane == 0) { sh.red[warp] = gt; sh.red2[warp] = eq; }
  __syncthreads();
  if (warp == 0) {
    const int g = __reduce_add_sync(0xffffffffu, lane < kTopWarps ? sh.red[lane] : 0u), e = __reduce_add_sync(0xffffffffu, lane < kTopWarps ? sh.red2[lane] : 0u);
    if (lane == 0) { sh.part[ex][0] = g; sh.part[ex][1] = e; }
  }
  cl.sync();
  int at_gt = 0, at_eq = 0;
  for (int q = 0; q < rank; ++q) { const TopShared* o = cl.map_shared_rank(&sh, q); at_gt += o->part[ex][0]; at_eq += o->part[ex][1]; }
  for (int q = 0; q < warp; ++q) { at_gt += sh.red[q]; at_eq += sh.red2[q]; }
  for (int i0 = s0; i0 < s1; i0 += 32) {
    const int i = i0 + lane;
    const uint32_t k = i < s1 ? key_at(i) : 0u;
    const uint32_t mg = __ballot_sync(0xffffffffu, i < s1 && k > cut), me = __ballot_sync(0xffffffffu, i < s1 && k == cut);
    const uint32_t below = (1u << lane) - 1;
    const int e = at_eq + __popc(me & below);
    const bool take = i < s1 && (k > cut || (k == cut && e < static_cast<int>(ties)));
    const int o = at_gt + __popc(mg & below) + min(e, static_cast<int>(ties));
    if (take && o < top_k) out[o] = base + i;
    at_gt += __popc(mg);
    at_eq += __popc(me);
  }
  cl.sync();                              // other CTAs may still read this one's words
}

// One warp per (query row, selected slot): copies the selected token's latent-cache row (row_bytes) and scale into
// the row's compact cache, whose pages the dense decode kernel then walks; the per-page scale bound is kept with an
// integer atomic max (scales are positive floats).  Unselected slots (-1) are left alone: the compact length hides them.
__global__ void dsa_gather_kernel(uint8_t* ckv, float* cscale, float* csmax, int* clen, const int* sel, int top_k,
                                  const uint8_t* cache, const float* scale, const int* pos, const int* seq,
                                  const int* page_table, int max_pages, int rows, int row_bytes) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + wib;
  if (item >= static_cast<long long>(rows) * top_k) return;
  const int r = static_cast<int>(item / top_k), j = static_cast<int>(item % top_k);
  if (j == 0 && lane == 0) clen[r] = max(0, min(pos[r] + 1, top_k));
  const int t = sel[item];
  if (t < 0) return;
  const int page = page_table[static_cast<size_t>(seq[r]) * max_pages + t / kIdxPage];
  const size_t src = static_cast<size_t>(page) * kIdxPage + t % kIdxPage;
  const size_t dst = static_cast<size_t>(r) * top_k + j;                 // compact pages are contiguous per row
  const uint4* s4 = reinterpret_cast<const uint4*>(cache + src * row_bytes);
  uint4* d4 = reinterpret_cast<uint4*>(ckv + dst * row_bytes);
  for (int u = lane; u < row_bytes / 16; u += 32) d4[u] = s4[u];
  if (lane == 0) {
    const float sc = scale[src];
    cscale[dst] = sc;
    atomicMax(reinterpret_cast<int*>(csmax + (dst / kIdxPage) * 4), __float_as_int(sc));
  }
}

}  // namespace plow

extern "C" {

// k bf16 [rows][ld_k] (128 index dims); cache e4m3 [n_pages][64][128]; cache_scale f32 [n_pages][64].
int plow_dsa_k_write(void* cache, float* cache_scale, const void* k, int ld_k, const float* gamma, const float* beta,
                     const float* rope_tab, const int* pos, const int* seq, const int* page_table, int max_pages,
                     int rows, int rot, int pair_mode, float eps, void* stream) {
  using namespace plow;
  if (rows <= 0 || rot > kIdxDim || rot % 2) return -1;
  plow::launch_serial(dsa_k_write_kernel, dim3((rows + 7) / 8), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 
      static_cast<uint8_t*>(cache), cache_scale, static_cast<const __nv_bfloat16*>(k), ld_k, gamma, beta, rope_tab, pos, seq,
      page_table, max_pages, rows, rot, pair_mode, eps);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

// q bf16 [rows][ld_q] (64 heads x 128); w f32 [rows][ld_w] head weights; scratch q8 e4m3 [rows][64][128], wq f32 [rows][64];
// scores f32 [rows][ld_scores] (scratch, ld_scores >= max visible length); sel int32 [rows][top_k].
int plow_dsa_select(int* sel, float* scores, int ld_scores, void* q8, float* wq, const void* q, int ld_q, const float* w,
                    int ld_w, const void* cache, const float* cache_scale, int64_t n_pages, const float* rope_tab,
                    const int* pos, const int* seq, const int* page_table, int max_pages, int rows, int rot, int pair_mode,
                    int top_k, int max_len, int* status, void* stream_) {
  using namespace plow;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (rows <= 0 || top_k <= 0 || max_len <= 0 || max_len > ld_scores || max_len > (1 << 20)) return -1;
  plow::launch_serial(dsa_q_prep_kernel, dim3((rows * kIdxHeads + 7) / 8), dim3(256), 0, stream, static_cast<uint8_t*>(q8), wq, static_cast<const __nv_bfloat16*>(q),
                                                                    ld_q, w, ld_w, rope_tab, pos, rows, rot, pair_mode);
  CUtensorMap tk, tq;
  int rc = make_tmap_2d(&tk, cache, 1, static_cast<uint64_t>(n_pages) * kIdxPage, kIdxDim, kIdxDim, kIdxPage, 128);
  if (rc) return 1100 + rc;
  rc = make_tmap_2d(&tq, q8, 1, static_cast<uint64_t>(rows) * kIdxHeads, kIdxDim, kIdxDim, kIdxHeads, 128);
  if (rc) return 1200 + rc;
  static DeviceOnce attr;
  if (ensure_smem(attr, dsa_score_kernel, kScoreSmem) != cudaSuccess) return 3000;
  // tiles per CTA: as few as still fit the chip at once (three CTAs per SM).  A CTA takes its tiles one after the other: 8 rows of 1500
  // tokens took 19.5 us at eight tiles, 15.3 at one.
  const int tiles = (max_len + 127) / 128;
  int per = kScoreTiles;
  while (per > 1 && static_cast<long long>(rows) * ((2 * tiles + per - 1) / per) <= 3 * sm_count()) per >>= 1;
  plow::launch_serial(dsa_score_kernel, dim3((tiles + per - 1) / per, rows), dim3(160), kScoreSmem, stream, scores, ld_scores, per, wq, cache_scale, pos, seq, page_table, max_pages, status, tk, tq);
  // CTAs per row: while the rows alone leave SMs idle or a CTA would hold over a quarter of its room (two to four stay
  // resident per SM), but none with under 1024 elements, where the cluster's barriers cost more than the passes
  int nc = 1;
  while (nc < kTopCluster && ((max_len + nc - 1) / nc > kTopSlice / 4 || static_cast<long long>(rows) * nc < 2 * sm_count()) && max_len / (2 * nc) >= 1024) nc <<= 1;
  const int slice = ((max_len + nc - 1) / nc + 31) & ~31;
  const int slice_cap = slice <= kTopSlice ? slice : 0;
  static DeviceOnce attr2;
  if (ensure_smem(attr2, dsa_topk_kernel, static_cast<int>(4 * (kTopBins + kTopCap + kTopSlice))) != cudaSuccess) return 3000;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * nc);
  cfg.blockDim = dim3(kTopThreads);
  cfg.dynamicSmemBytes = 4 * static_cast<size_t>(kTopBins + kTopCap + slice_cap);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nc; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, dsa_topk_kernel, sel, static_cast<const float*>(scores), ld_scores, pos, top_k, slice_cap);
  if (le != cudaSuccess) return 4000 + static_cast<int>(le);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

// Gather the selected cache rows of every query row into its compact cache: ckv [rows*top_k/64 pages][64][row_bytes],
// cscale f32 [pages][64], csmax f32 [pages][4] (zeroed here), clen int32 [rows] = min(pos+1, top_k).  top_k % 64 == 0.
int plow_dsa_gather(void* ckv, float* cscale, float* csmax, int* clen, const int* sel, int top_k, const void* cache,
                    const float* scale, const int* pos, const int* seq, const int* page_table, int max_pages, int rows,
                    int row_bytes, void* stream_) {
  using namespace plow;
  if (rows <= 0 || top_k <= 0 || top_k % kIdxPage || row_bytes % 16) return -1;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  const size_t pages = static_cast<size_t>(rows) * (top_k / kIdxPage);
  cudaMemsetAsync(csmax, 0, pages * 4 * sizeof(float), stream);
  const long long items = static_cast<long long>(rows) * top_k;
  plow::launch_serial(dsa_gather_kernel, dim3(static_cast<unsigned>((items + 7) / 8)), dim3(256), 0, stream, 
      static_cast<uint8_t*>(ckv), cscale, csmax, clen, sel, top_k, static_cast<const uint8_t*>(cache), scale, pos, seq,
      page_table, max_pages, rows, row_bytes);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

}  // extern "C"
