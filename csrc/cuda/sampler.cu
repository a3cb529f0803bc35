// Device sampler: temperature -> top-k -> softmax -> top-p -> min-p -> renormalise -> inverse-CDF draw, entirely in
// f32 over the row's logits.  Ties at a cut value are all kept.  Rows whose temperature is <= 0 take the arg-max
// (lowest index on ties).  The filter order is the host sampler's (plow_b200/text/sample.py); reference:
// runtime/nvidia/sample_sm120.cu, crates/plowrt/src/text/sample.rs.  The uniform variate comes from the caller (u[row])
// or, when u is NULL, from a counter hash of (seed[row], step) so a request with a seed replays identically.
//
// One thread-block cluster per row.  The row is read from HBM once; every CTA keeps its contiguous slice of the scaled
// logits in shared memory and all later passes run there, partial results crossing the cluster through distributed
// shared memory.  (One 1024-thread CTA per row that re-read the row for each of up to twelve passes and counted into one
// shared histogram with atomics took 2620 us for 256 rows x 128256: the leading digit of the logits hits a handful of
// counters, and shared f32 atomics are compare-and-swap loops.)
//
// The cut of a filter - the largest key T such that weight({key >= T}) >= target, weight = element count for top-k,
// probability mass for top-p - is found by narrowing: 16 bins of the distance to the maximum (later: of the key range of
// the bin that holds the cut), each thread owning one private counter per bin, so there are no atomics and the sums are
// the same on every run; when the bin that holds the cut has at most kCap elements they are gathered into the first
// CTA's shared memory and sorted.  A top-k row whose candidates fit there altogether is finished in that list.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include "launch.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kBins = 16;                // = kWarps: warp b sums bin b
constexpr int kCap = 2048;               // elements of the gathered list
constexpr int kMaxCluster = 8;
// Slice of a row a CTA keeps in shared memory: with the bins 110 KB, so two CTAs share an SM and one loads while the
// other one counts.  Wider rows take up to kSliceMax (one CTA per SM), wider still are re-read from global memory.
constexpr int kSlice = 19456;
constexpr int kSliceMax = 45056;

static_assert(kBins == kWarps, "one warp per bin");

__device__ __forceinline__ uint32_t ordered_key(float x) {   // monotone: larger float -> larger key
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

__device__ __forceinline__ float hash_uniform(unsigned long long seed, unsigned long long ctr) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (ctr + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return static_cast<float>(z >> 40) * (1.0f / 16777216.0f);   // [0, 1)
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_incl(float v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Static shared memory of a CTA.  `part` carries a CTA's share of a cluster-wide result; two buffers in turn, so that one
// cluster barrier per exchange is enough (a buffer is rewritten only after the barrier of the exchange in between).
struct Shared {
  union { float f; uint32_t u; } part[2][kWarps];
  float red[kWarps];
  int cnt[kWarps];
  float bc_f;
  int bc_i;
};

struct Row {
  __device__ static cg::cluster_group cl() { return cg::this_cluster(); }
  Shared* sh;
  float* xs;            // slice of scaled logits (in_smem) or unused
  float* bins;          // [kBins][kThreads] private counters; the gathered list of the first CTA lies over them
  const float* lg;      // the slice in global memory
  float invT;
  int n, base;          // elements of the slice, vocabulary index of its first one
  int nc, rank;
  bool in_smem;
  int ex;               // exchange parity
  int tid, lane, warp;
  int seg0, seg1;       // this warp's contiguous part of the slice

  __device__ float x(int i) const { return in_smem ? xs[i] : lg[i] * invT; }
  __device__ Shared* peer(int r) { return cl().map_shared_rank(sh, r); }
  // this CTA's part values are in part[ex]; afterwards every CTA may read all of them
  __device__ int exchange() { cl().sync(); const int b = ex; ex ^= 1; return b; }

  __device__ float sum_all(float v) {
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sh->red[warp] = v;
    __syncthreads();
    if (tid == 0) { float s = 0.f; for (int w = 0; w < kWarps; ++w) s += sh->red[w]; sh->part[ex][0].f = s; }
    const int b = exchange();
    float s = 0.f;
    for (int r = 0; r < nc; ++r) s += peer(r)->part[b][0].f;
    return s;
  }
};

// Bins (descending: bin 0 holds the largest keys) of the elements that can still hold the cut.
struct Interval {
  float mx;
  int b0;                 // -1: the sixteen unit-wide bins of mx - x; else: elements of that bin with keys in [klo, khi]
  uint32_t klo, khi, step;
  __device__ int bin0(float x) const { return static_cast<int>(fminf(mx - x, 15.0f)); }      // NaN counts as far away
  __device__ int bin(float x) const {
    const int b = bin0(x);
    if (b0 < 0) return b;
    if (b != b0) return -1;
    const uint32_t k = ordered_key(x);
    return (k < klo || k > khi) ? -1 : static_cast<int>((khi - k) / step);
  }
  __device__ void set_step() { const uint32_t w = khi - klo; step = w / kBins + 1; }
  // narrow to bin s
  __device__ void enter(int s) {
    if (b0 < 0) {
      b0 = s;
      // edges of the unit bin with slack for the rounding of mx - x; the last bin is open
      const float slack = 1e-6f * (fabsf(mx) + 16.0f);
      khi = ordered_key(mx - static_cast<float>(s) + slack);
      klo = s >= kBins - 1 ? 0u : ordered_key(mx - static_cast<float>(s + 1) - slack);
      if (s == 0) khi = 0xFFFFFFFFu;
    } else {
      khi -= min(static_cast<uint32_t>(s), (khi - klo) / step) * step;
      klo = khi - klo >= step - 1 ? khi - (step - 1) : klo;
    }
    set_step();
  }
  __device__ bool single() const { return b0 >= 0 && klo == khi; }
  __device__ bool inside(float x) const {
    const int b = bin0(x);
    if (b0 < 0) return true;
    if (b != b0) return false;
    const uint32_t k = ordered_key(x);
    return k >= klo && k <= khi;
  }
  // inside, or larger than everything inside
  __device__ bool reached(float x) const {
    const int b = bin0(x);
    return b0 < 0 || b < b0 || (b == b0 && ordered_key(x) >= klo);
  }
};

// One counting pass over the interval.  Returns the bin that holds the cut, adds the weight of the bins before it to
// `above` and leaves the bin's own weight in `own`.  A target that is not reached gives kBins for the whole row, and the
// last bin that holds anything for a narrower interval (the sums of another order fell short by a rounding).
template <class Weight>
__device__ int find_bin(Row& r, const Interval& iv, float target, float& above, float& own, Weight weight) {
  __syncthreads();
#pragma unroll
  for (int b = 0; b < kBins; ++b) r.bins[b * kThreads + r.tid] = 0.f;
  for (int i = r.tid; i < r.n; i += kThreads) {
    const float x = r.x(i);
    const int b = iv.bin(x);
    if (b >= 0) r.bins[b * kThreads + r.tid] += weight(x);
  }
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < kThreads / 32; ++j) s += r.bins[r.warp * kThreads + j * 32 + r.lane];
  s = warp_sum(s);
  if (r.lane == 0) r.sh->part[r.ex][r.warp].f = s;
  const int buf = r.exchange();
  float h = 0.f;                                    // lane b: weight of bin b over the cluster
  if (r.lane < kBins)
    for (int q = 0; q < r.nc; ++q) h += r.peer(q)->part[buf][r.lane].f;
  int last = kBins;
  float acc = above, last_above = above;
  for (int b = 0; b < kBins; ++b) {
    const float hb = __shfl_sync(0xffffffffu, h, b);
    if (acc + hb >= target) { above = acc; own = hb; return b; }
    if (hb > 0.f && iv.b0 >= 0) { last = b; last_above = acc; own = hb; }
    acc += hb;
  }
  above = last_above;
  return last;
}

// Gathers the elements that satisfy `pred` into the list of the first CTA (its own `bins` memory: x, then the vocabulary
// index), in index order.  Returns how many there are; more than kCap are counted and not written.
template <class Pred>
__device__ int gather(Row& r, Pred pred) {
  int c = 0;
  for (int i = r.seg0; i < r.seg1; i += 32) {
    const bool in = i + r.lane < r.seg1 && pred(r.x(i + r.lane));
    c += __popc(__ballot_sync(0xffffffffu, in));
  }
  __syncthreads();
  if (r.lane == 0) { r.sh->cnt[r.warp] = c; r.sh->part[r.ex][r.warp].u = static_cast<uint32_t>(c); }
  const int buf = r.exchange();                     // also: no CTA still reads the memory under the list
  int at = 0, total = 0;
  for (int q = 0; q < r.nc; ++q) {
    const Shared* p = r.peer(q);
    const int v = r.lane < kWarps ? static_cast<int>(p->part[buf][r.lane].u) : 0;
    const int all = __reduce_add_sync(0xffffffffu, v);
    if (q < r.rank) at += all;
    total += all;
  }
  if (total > kCap) return total;
  for (int w = 0; w < r.warp; ++w) at += r.sh->cnt[w];
  float* lx = r.cl().map_shared_rank(r.bins, 0);
  int* li = reinterpret_cast<int*>(lx + kCap);
  for (int i = r.seg0; i < r.seg1; i += 32) {
    const float x = i + r.lane < r.seg1 ? r.x(i + r.lane) : 0.f;
    const bool in = i + r.lane < r.seg1 && pred(x);
    const uint32_t m = __ballot_sync(0xffffffffu, in);
    if (in) {
      const int o = at + __popc(m & ((1u << r.lane) - 1));
      lx[o] = x;
      li[o] = r.base + i + r.lane;
    }
    at += __popc(m);
  }
  return total;
}

// In-place descending bitonic sort of n2 (a power of two) keys by one CTA.
__device__ void sort_desc(uint32_t* k, int n2, int tid) {
  for (int size = 2; size <= n2; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int t = tid; t < n2 / 2; t += kThreads) {
        const int i = 2 * t - (t & (stride - 1)), j = i + stride;
        const uint32_t a = k[i], b = k[j];
        if ((a < b) == ((i & size) == 0)) { k[i] = b; k[j] = a; }
      }
    }
  __syncthreads();
}

// Keys of the gathered list, sorted descending and padded with zeros, behind the list.  First CTA only.
__device__ uint32_t* sorted_list(Row& r, int n) {
  uint32_t* sk = reinterpret_cast<uint32_t*>(r.bins) + 2 * kCap;
  static_assert(3 * kCap <= kBins * kThreads, "list and sorted keys lie over the bins");
  int n2 = 32;
  while (n2 < n) n2 <<= 1;
  for (int i = r.tid; i < n2; i += kThreads) sk[i] = i < n ? ordered_key(r.bins[i]) : 0u;
  sort_desc(sk, n2, r.tid);
  return sk;
}

// Exclusive prefix of v over the CTA's threads; *total receives the sum.
__device__ float block_excl(Row& r, float v, float* total) {
  const float incl = warp_incl(v, r.lane);
  __syncthreads();
  if (r.lane == 31) r.sh->red[r.warp] = incl;
  __syncthreads();
  float base = 0.f, all = 0.f;
  for (int w = 0; w < kWarps; ++w) { if (w < r.warp) base += r.sh->red[w]; all += r.sh->red[w]; }
  *total = all;
  return base + incl - v;
}

// First position of the sorted keys at which `above` plus the prefix of their masses reaches the target.  First CTA only.
template <class Weight>
__device__ int first_reaching(Row& r, const uint32_t* sk, int n, float above, float target, Weight weight) {
  constexpr int kPer = kCap / kThreads;
  float w[kPer], local = 0.f, all;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = r.tid * kPer + j;
    w[j] = i < n ? weight(key_value(sk[i])) : 0.f;
    local += w[j];
  }
  float acc = above + block_excl(r, local, &all);
  if (r.tid == 0) r.sh->bc_i = n - 1;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    acc += w[j];
    if (r.tid * kPer + j < n && acc >= target) { atomicMin(&r.sh->bc_i, r.tid * kPer + j); break; }
  }
  __syncthreads();
  const int pos = r.sh->bc_i;
  __syncthreads();
  return pos;
}

__global__ void __launch_bounds__(kThreads)
sample_kernel(int* out, const float* logits, int ld, int V, int slice, int in_smem, const float* temperature, const int* top_k,
              const float* top_p, const float* min_p, const float* u_in, const unsigned long long* seed,
              unsigned long long step) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  extern __shared__ __align__(16) float dyn[];
  __shared__ Shared sh;
  Row r;

  r.sh = &sh;
  r.nc = static_cast<int>(r.cl().num_blocks());
  r.rank = static_cast<int>(r.cl().block_rank());
  r.tid = threadIdx.x; r.lane = threadIdx.x & 31; r.warp = threadIdx.x >> 5;
  const int row = blockIdx.x / r.nc;
  r.base = min(V, r.rank * slice);
  r.n = min(V, r.base + slice) - r.base;
  r.bins = dyn;
  r.xs = dyn + kBins * kThreads;
  r.in_smem = in_smem != 0;
  r.ex = 0;
  const int seg = ((r.n + kWarps - 1) / kWarps + 31) & ~31;
  r.seg0 = min(r.n, r.warp * seg);
  r.seg1 = min(r.n, r.seg0 + seg);
  const float* lg = logits + static_cast<size_t>(row) * ld + r.base;
  r.lg = lg;
  const float T = temperature ? temperature[row] : 1.0f;
  if (T <= 0.f) {
    // arg-max, lowest index on ties: packed (ordered value, ~index)
    unsigned long long best = 0;
#pragma unroll 8
    for (int i = r.tid; i < r.n; i += kThreads) {
      const unsigned long long k = (static_cast<unsigned long long>(ordered_key(lg[i])) << 32) | (0xFFFFFFFFu - (r.base + i));
      best = k > best ? k : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
      best = t > best ? t : best;
    }
    __shared__ unsigned long long bw[kWarps];
    if (r.lane == 0) bw[r.warp] = best;
    __syncthreads();
    if (r.tid == 0) {
      for (int w = 1; w < kWarps; ++w) best = bw[w] > best ? bw[w] : best;
      bw[0] = best;
    }
    r.cl().sync();
    if (r.rank == 0 && r.tid == 0) {
      for (int q = 1; q < r.nc; ++q) {
        const unsigned long long t = *r.cl().map_shared_rank(bw, q);
        best = t > best ? t : best;
      }
      out[row] = static_cast<int>(0xFFFFFFFFu - static_cast<uint32_t>(best & 0xFFFFFFFFu));
    }
    r.cl().sync();        // the other CTAs' words stay readable until here
    return;
  }
  const float invT = r.invT = 1.0f / fmaxf(T, 1e-6f);
  float mx = -INFINITY;
  if (r.in_smem) {
    if (((reinterpret_cast<uintptr_t>(lg) & 15) | (r.n & 3)) == 0) {
#pragma unroll 4
      for (int i = r.tid; i < r.n / 4; i += kThreads) {
        float4 v = reinterpret_cast<const float4*>(lg)[i];
        v.x *= invT; v.y *= invT; v.z *= invT; v.w *= invT;
        reinterpret_cast<float4*>(r.xs)[i] = v;
        mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
      }
    } else {
#pragma unroll 8
      for (int i = r.tid; i < r.n; i += kThreads) { const float v = lg[i] * invT; r.xs[i] = v; mx = fmaxf(mx, v); }
    }
  } else {
#pragma unroll 8
    for (int i = r.tid; i < r.n; i += kThreads) mx = fmaxf(mx, lg[i] * invT);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (r.lane == 0) sh.part[r.ex][r.warp].f = mx;
  {
    const int buf = r.exchange();
    mx = -INFINITY;
    for (int q = 0; q < r.nc; ++q) mx = fmaxf(mx, r.lane < kWarps ? r.peer(q)->part[buf][r.lane].f : -INFINITY);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  const float u = u_in ? u_in[row] : hash_uniform(seed ? seed[row] : 0ull, step);
  const float tp = top_p ? top_p[row] : 1.0f;
  const bool nucleus = tp < 1.0f && tp > 0.f;      // a target of zero keeps everything
  const float mp = min_p ? min_p[row] : 0.f;
  uint32_t k_key = 0;                              // key of the k-th largest scaled logit
  const int k = top_k ? top_k[row] : 0;
  if (k > 0 && k < V) {
    Interval iv{mx, -1, 0u, 0u, 1u};
    float above = 0.f, own = 0.f;
    const float kf = static_cast<float>(k);
    auto one = [](float) { return 1.0f; };
    int cut = find_bin(r, iv, kf, above, own, one);
    iv.enter(min(cut, kBins - 1));
    while (own > 0.f && !iv.single() && (k <= kCap ? above + own > kCap : own > kCap)) {
      cut = find_bin(r, iv, kf, above, own, one);
      iv.enter(min(cut, kBins - 1));
    }
    if (k <= kCap && above + own <= kCap) {
      // every candidate fits the list: the first CTA finishes the row there
      const int n = gather(r, [&](float x) { return iv.reached(x); });
      r.cl().sync();
      if (r.rank == 0) {
        const uint32_t* sk = sorted_list(r, n);
        k_key = sk[min(k, n) - 1];
        const float* lx = r.bins;
        const int* li = reinterpret_cast<const int*>(r.bins + kCap);
        auto e_of = [&](float x) { return ordered_key(x) >= k_key ? __expf(x - mx) : 0.f; };
        constexpr int kPer = kCap / kThreads;
        float e[kPer], local = 0.f, z;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          const int i = r.tid * kPer + j;
          e[j] = i < n ? e_of(lx[i]) : 0.f;
          local += e[j];
        }
        block_excl(r, local, &z);
        const float invZ = 1.0f / z;
        float p_cut = 0.f;
        if (nucleus) {
          const int pos = first_reaching(r, sk, n, 0.f, tp, [&](float x) { return e_of(x) * invZ; });
          p_cut = e_of(key_value(sk[pos])) * invZ;
        }
        p_cut = fmaxf(p_cut, mp * invZ);             // the largest probability is exp(0) / Z
        local = 0.f;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          const float p = e[j] * invZ;
          e[j] = (p >= p_cut && p > 0.f) ? p : 0.f;
          local += e[j];
        }
        float total;
        const float lo = block_excl(r, local, &total);
        const float target = u * total;
        // the first kept index whose running sum passes the target; rounding at the end: the last kept index
        if (r.tid == 0) { sh.bc_i = INT_MAX; sh.cnt[0] = -1; }
        __syncthreads();
        float acc = lo;
        int last = -1;
        bool hit = false;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          if (e[j] > 0.f) {
            last = r.tid * kPer + j;
            acc += e[j];
            if (!hit && target < acc) { hit = true; atomicMin(&sh.bc_i, last); }
          }
        }
        if (last >= 0) atomicMax(&sh.cnt[0], last);
        __syncthreads();
        if (r.tid == 0) {
          const int at = sh.bc_i != INT_MAX ? sh.bc_i : sh.cnt[0];
          out[row] = at >= 0 ? li[at] : -1;
        }
      }
      return;           // nobody reads another CTA's memory after the barrier above
    }
    if (iv.single()) {
      k_key = iv.klo;
    } else {
      const int n = gather(r, [&](float x) { return iv.inside(x); });
      r.cl().sync();
      if (r.rank == 0) {
        const int at = min(n - 1, max(0, k - static_cast<int>(above) - 1));
        const uint32_t* sk = sorted_list(r, n);
        if (r.tid == 0) sh.bc_i = static_cast<int>(n > 0 ? sk[at] : 0u);
      }
      r.cl().sync();
      k_key = static_cast<uint32_t>(r.peer(0)->bc_i);
      r.cl().sync();
    }
  }
  auto e_of = [&](float x) -> float { return ordered_key(x) >= k_key ? __expf(x - mx) : 0.f; };
  float z = 0.f;
#pragma unroll 4
  for (int i = r.tid; i < r.n; i += kThreads) z += e_of(r.x(i));
  z = r.sum_all(z);
  const float invZ = 1.0f / z;
  auto mass = [&](float x) { return e_of(x) * invZ; };
  // top-p: smallest set of the largest probabilities whose mass reaches top_p
  float p_cut = 0.f;
  if (nucleus) {
    Interval iv{mx, -1, 0u, 0u, 1u};
    float above = 0.f, own = 0.f;
    int cut = find_bin(r, iv, tp, above, own, mass);
    if (cut < kBins) {
      iv.enter(cut);
      int n;
      // a unit-wide bin of mass `own` holds at least own / (its largest probability) elements: skip a gather that cannot fit
      const float most = __expf(-static_cast<float>(cut)) * invZ;
      bool deeper = own > most * kCap;
      while (true) {
        if (iv.single()) { n = 0; break; }
        if (!deeper) {
          n = gather(r, [&](float x) { return iv.inside(x); });
          if (n <= kCap) break;
        }
        deeper = false;
        cut = find_bin(r, iv, tp, above, own, mass);
        iv.enter(min(cut, kBins - 1));
      }
      if (iv.single()) {
        p_cut = mass(key_value(iv.klo));
      } else {
        r.cl().sync();
        if (r.rank == 0) {
          const uint32_t* sk = sorted_list(r, n);
          const int pos = n > 0 ? first_reaching(r, sk, n, above, tp, mass) : 0;
          if (r.tid == 0) sh.bc_f = n > 0 ? mass(key_value(sk[pos])) : 0.f;
        }
        r.cl().sync();
        p_cut = r.peer(0)->bc_f;
        r.cl().sync();
      }
    }
  }
  p_cut = fmaxf(p_cut, mp * invZ);               // the largest probability is exp(0) / Z
  auto p_of = [&](float x) -> float {
    const float p = mass(x);
    return (p >= p_cut && p > 0.f) ? p : 0.f;
  };
  // inverse CDF in index order: sums of the warps' contiguous parts, then the warp whose part holds the target walks it
  float ps = 0.f;
  for (int i = r.seg0 + r.lane; i < r.seg1; i += 32) ps += p_of(r.x(i));
  ps = warp_sum(ps);
  if (r.lane == 0) sh.part[r.ex][r.warp].f = ps;
  const int buf = r.exchange();
  float total = 0.f;
  for (int q = 0; q < r.nc; ++q) {
    const float v = r.lane < kWarps ? r.peer(q)->part[buf][r.lane].f : 0.f;
    for (int w = 0; w < kWarps; ++w) total += __shfl_sync(0xffffffffu, v, w);
  }
  const float target = u * total;
  float acc = 0.f, own_lo = 0.f;
  int at = -1, last = -1;          // global part number that holds the target; last part that keeps anything
  float last_lo = 0.f;
  for (int q = 0; q < r.nc; ++q) {
    const float v = r.lane < kWarps ? r.peer(q)->part[buf][r.lane].f : 0.f;
    for (int w = 0; w < kWarps; ++w) {
      const float s = __shfl_sync(0xffffffffu, v, w);
      if (s > 0.f) {
        last = q * kWarps + w; last_lo = acc;
        if (at < 0 && target < acc + s) { at = last; own_lo = acc; }
        acc += s;
      }
    }
  }
  if (at < 0) { at = last; own_lo = last_lo; }
  if (at < 0) {
    if (r.rank == 0 && r.tid == 0) out[row] = -1;
  } else if (at == r.rank * kWarps + r.warp) {
    float run = own_lo;
    int pick = -1, kept = -1;
    for (int i = r.seg0; i < r.seg1 && pick < 0; i += 32) {
      const float p = i + r.lane < r.seg1 ? p_of(r.x(i + r.lane)) : 0.f;
      const float incl = warp_incl(p, r.lane);
      const uint32_t any = __ballot_sync(0xffffffffu, p > 0.f);
      const uint32_t hit = __ballot_sync(0xffffffffu, p > 0.f && target < run + incl);
      if (any) kept = i + 31 - __clz(any);
      if (hit) pick = i + __ffs(hit) - 1;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (pick < 0) pick = kept;     // rounding left the target at or past the part's end: its last kept index
    if (r.lane == 0) out[row] = pick >= 0 ? r.base + pick : -1;
  }
  r.cl().sync();                     // other CTAs may still read this one's sums
}

}  // namespace

extern "C" {

// logits f32 [rows][ld]; temperature / top_p / min_p f32 [rows] and top_k int32 [rows] (each may be NULL =
// neutral); u f32 [rows] uniform variates in [0,1) or NULL to hash (seed[row], step); out int32 [rows].
int plow_sample(int* out, const float* logits, int ld, int rows, int V, const float* temperature, const int* top_k,
                const float* top_p, const float* min_p, const float* u, const void* seed, uint64_t step, void* stream) {
  if (rows <= 0 || V <= 0) return -1;
  // CTAs per row: as many as it takes for the slices to fit two CTAs to an SM, and while the rows alone leave SMs idle
  // up to eight (a slice is not cut below 1024 elements); both ends measured, see above.
  int nc = 1;
  while (nc < kMaxCluster && (V + nc - 1) / nc > kSlice) nc <<= 1;
  while (nc < kMaxCluster && static_cast<long long>(rows) * nc < 2 * 148 && V / (2 * nc) >= 1024) nc <<= 1;
  const int slice = ((V + nc - 1) / nc + 3) & ~3;
  const int in_smem = slice <= kSliceMax;
  const size_t smem = sizeof(float) * (kBins * kThreads + (in_smem ? slice : 0));
  static plow::DeviceOnce attr;
  if (plow::ensure_smem(attr, sample_kernel, static_cast<int>(sizeof(float) * (kBins * kThreads + kSliceMax))) != cudaSuccess) return 3000;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * nc);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nc; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, sample_kernel, out, logits, ld, V, slice, in_smem, temperature, top_k, top_p, min_p, u,
                                     static_cast<const unsigned long long*>(seed), static_cast<unsigned long long>(step));
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

}  // extern "C"
