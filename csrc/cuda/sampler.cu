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
// counters, and shared f32 atomics are compare-and-swap loops.  This kernel: 213 us, 15 to 19 us for one
// unfiltered row of 32000 or 128256.  It is bound by the chain of passes, not by memory: reading the logits alone takes 20 us, DRAM is
// 6 % and issue slots are 43 % busy, and the longest stalls are at the barriers of the CTAs and clusters.)
//
// The cut of a filter - the largest key T such that weight({key >= T}) >= target, weight = element count for top-k,
// probability mass for top-p - is found by narrowing: 16 bins of the distance to the maximum (later: of the key range of
// the bin that holds the cut), each thread owning one private counter per bin, so there are no atomics and the sums are
// the same on every run; when the bin that holds the cut has at most kCap elements they are gathered into the first
// CTA's shared memory and sorted.  A top-k row whose candidates fit there altogether is finished in that list.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <stdint.h>

#include "launch.cuh"
#include "tmap.cuh"

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

// largest of three, NaN if any is one: one such logit leaves the row without probabilities
__device__ __forceinline__ float max_nan(float a, float b, float c) { float r; asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float max_nan(float a, float b) { return max_nan(a, b, b); }

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
  float bc_f;
  int bc_i, last;
};

struct Row {
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
  int seg0, seg1;       // this warp's contiguous part of the slice (seg0 a multiple of 128)

  __device__ static cg::cluster_group cl() { return cg::this_cluster(); }
  __device__ float x(int i) const { return in_smem ? xs[i] : lg[i] * invT; }
  __device__ Shared* peer(int r) { return cl().map_shared_rank(sh, r); }
  // this CTA's part values are in part[ex]; afterwards every CTA may read all of them
  __device__ int exchange() { sync(); const int b = ex; ex ^= 1; return b; }
  __device__ void sync() const { if (nc > 1) cl().sync(); else __syncthreads(); }

  // f(x) for every element of the slice, four at a time from shared memory
  template <class F>
  __device__ void each(F f) const {
    if (in_smem) {
#pragma unroll 2
      for (int i = tid; i < n / 4; i += kThreads) {
        const float4 v = reinterpret_cast<const float4*>(xs)[i];
        f(v.x); f(v.y); f(v.z); f(v.w);
      }
      if (tid < (n & 3)) f(xs[(n & ~3) + tid]);
    } else {
      for (int i = tid; i < n; i += kThreads) f(lg[i] * invT);
    }
  }
  // f(x) for every element of this warp's part; the warp's lanes see different ones
  template <class F>
  __device__ void each_of_part(F f) const {
    int i = seg0 + 4 * lane;
    if (in_smem) {
#pragma unroll 2
      for (; i + 4 <= seg1; i += 128) {
        const float4 v = *reinterpret_cast<const float4*>(xs + i);
        f(v.x); f(v.y); f(v.z); f(v.w);
      }
      for (; i < seg1; ++i) f(xs[i]);        // at most one lane, fewer than four elements
    } else {
      for (i = seg0 + lane; i < seg1; i += 32) f(lg[i] * invT);
    }
  }
  // four consecutive elements from i (a multiple of 4) of this warp's part; missing ones are NaN and not ok
  __device__ float4 quad(int i, int* count) const {
    const float nan = __int_as_float(0x7fffffff);
    const int c = min(4, max(0, seg1 - i));
    *count = c;
    if (c == 4 && in_smem) return *reinterpret_cast<const float4*>(xs + i);
    return make_float4(c > 0 ? x(i) : nan, c > 1 ? x(i + 1) : nan, c > 2 ? x(i + 2) : nan, c > 3 ? x(i + 3) : nan);
  }
};

// Bins (descending: bin 0 holds the largest elements) of what can still hold the cut.  The first level is sixteen unit-wide
// bins of the distance to the maximum; below it the key range of one bin is cut into sixteen.
struct Interval {
  float mx;
  int b0;                 // bin of the first level, -1 before it is known
  bool keyed;             // narrower than that bin: keys in [klo, khi]
  uint32_t klo, khi;
  int shift;              // a bin is 2^shift keys wide
  __device__ static Interval whole(float mx) { return Interval{mx, -1, false, 0u, 0u, 0}; }
  __device__ static int bin0(float d) { return static_cast<int>(fminf(d, 15.0f)); }      // NaN counts as far away
  __device__ bool in0(float d) const { return !(d < static_cast<float>(b0)) && (b0 == kBins - 1 || d < static_cast<float>(b0 + 1)); }
  __device__ int bin(float x) const {
    const float d = mx - x;
    if (b0 < 0) return bin0(d);
    const uint32_t k = ordered_key(x);
    return (!in0(d) || k < klo || k > khi) ? -1 : static_cast<int>((khi - k) >> shift);
  }
  // narrow to bin s
  __device__ void enter(int s) {
    if (b0 < 0) {
      b0 = s;
      // edges of the unit bin with slack for the rounding of mx - x; the last bin is open
      const float slack = 1e-6f * (fabsf(mx) + 16.0f);
      khi = s == 0 ? 0xFFFFFFFFu : ordered_key(mx - static_cast<float>(s) + slack);
      klo = s >= kBins - 1 ? 0u : ordered_key(mx - static_cast<float>(s + 1) - slack);
    } else {
      keyed = true;
      const uint32_t last = (1u << shift) - 1;
      khi -= min(static_cast<uint32_t>(s), (khi - klo) >> shift) << shift;
      klo = khi - klo >= last ? khi - last : klo;
    }
    shift = max(0, 28 - __clz(khi - klo));      // (khi - klo) >> shift < kBins
  }
  __device__ bool single() const { return keyed && klo == khi; }
  __device__ bool inside(float x) const {
    if (!in0(mx - x)) return false;
    const uint32_t k = ordered_key(x);
    return !keyed || (k >= klo && k <= khi);
  }
  // inside, or larger than everything inside
  __device__ bool reached(float x) const {
    const float d = mx - x;
    return d < static_cast<float>(b0) || (in0(d) && (!keyed || ordered_key(x) >= klo));
  }
};

// One counting pass over the interval.  Returns the bin that holds the cut, adds the weight of the bins before it to
// `above` and leaves the bin's own weight in `own`; `all` is the weight of all bins, `few` a lower bound on the number of
// elements in the bins up to the cut if a weight is the exponential of minus the distance.  The target is `share` of `all`
// where share > 0.  A target that is not reached gives kBins for the whole row, and the last bin that holds anything for a
// narrower interval (the sums of another order fell short by a rounding).
struct Cut { int bin; float all, few; };
template <class Weight>
__device__ Cut find_bin(Row& r, const Interval& iv, float target, bool share, float& above, float& own, Weight weight) {
  float* mine = r.bins + r.tid;
  __syncthreads();
#pragma unroll
  for (int b = 0; b < kBins; ++b) mine[b * kThreads] = 0.f;
  if (iv.b0 < 0)
    r.each([&](float x) { mine[Interval::bin0(iv.mx - x) * kThreads] += weight(x); });
  else
    r.each([&](float x) { const int b = iv.bin(x); if (b >= 0) mine[b * kThreads] += weight(x); });
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
  Cut c;
  c.all = warp_sum(h);
  if (share) target *= c.all;
  const float incl = above + warp_incl(h, r.lane);
  const uint32_t hit = __ballot_sync(0xffffffffu, r.lane < kBins && incl >= target);
  const uint32_t some = __ballot_sync(0xffffffffu, h > 0.f);
  c.bin = hit ? __ffs(hit) - 1 : (iv.b0 >= 0 && some ? 31 - __clz(some) : kBins);
  const float few = warp_incl(h * __expf(static_cast<float>(r.lane)), r.lane);
  const int at = min(c.bin, kBins - 1);
  c.few = __shfl_sync(0xffffffffu, few, at);
  own = __shfl_sync(0xffffffffu, h, at);
  const float before = __shfl_up_sync(0xffffffffu, incl, 1);
  above = at > 0 ? __shfl_sync(0xffffffffu, before, at) : above;
  return c;
}

// Gathers the elements that satisfy `pred` into the list of the first CTA (its own `bins` memory: x, then the vocabulary
// index), in index order.  Returns how many there are; more than kCap are counted and not written.
template <class Pred>
__device__ int gather(Row& r, Pred pred) {
  int c = 0, have;
  r.each_of_part([&](float x) { c += static_cast<int>(pred(x)); });
  c = __reduce_add_sync(0xffffffffu, c);
  __syncthreads();
  if (r.lane == 0) r.sh->part[r.ex][r.warp].u = static_cast<uint32_t>(c);
  const int buf = r.exchange();                     // also: no CTA still reads the memory under the list
  int at = 0, total = 0;
  for (int q = 0; q < r.nc; ++q) {
    const int v = r.lane < kWarps ? static_cast<int>(r.peer(q)->part[buf][r.lane].u) : 0;
    const int all = __reduce_add_sync(0xffffffffu, v);
    at += q < r.rank ? all : (q == r.rank ? __reduce_add_sync(0xffffffffu, r.lane < r.warp ? v : 0) : 0);
    total += all;
  }
  if (total > kCap) return total;
  float* lx = r.cl().map_shared_rank(r.bins, 0);
  int* li = reinterpret_cast<int*>(lx + kCap);
  if (c == 0) return total;
  for (int i0 = r.seg0; i0 < r.seg1; i0 += 128) {
    const int i = i0 + 4 * r.lane;
    const float4 v = r.quad(i, &have);
    const bool in[4] = {have > 0 && pred(v.x), have > 1 && pred(v.y), have > 2 && pred(v.z), have > 3 && pred(v.w)};
    const int mine = in[0] + in[1] + in[2] + in[3];
    if (!__any_sync(0xffffffffu, mine)) continue;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (r.lane >= o) incl += t;
    }
    int o = at + incl - mine;
    const float xv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (in[j]) { lx[o] = xv[j]; li[o] = r.base + i + j; ++o; }
    at += __shfl_sync(0xffffffffu, incl, 31);
  }
  return total;
}

// Keys of the gathered list, sorted descending and padded with zeros, behind the list.  First CTA only.  Bitonic, four
// consecutive keys per thread: strides below 4 stay in registers, below 128 in the warp (shuffles), only wider ones go
// through shared memory (a barrier per stage for every stride took 14k clocks for 1024 keys, this takes a quarter).
__device__ uint32_t* sorted_list(Row& r, int n) {
  uint32_t* sk = reinterpret_cast<uint32_t*>(r.bins) + 2 * kCap;
  static_assert(3 * kCap <= kBins * kThreads && kCap == 4 * kThreads, "list and sorted keys lie over the bins; four keys a thread");
  int n2 = 128;
  while (n2 < n) n2 <<= 1;
  uint32_t k[4];
  const int i0 = 4 * r.tid;
#pragma unroll
  for (int j = 0; j < 4; ++j) k[j] = i0 + j < n ? ordered_key(r.bins[i0 + j]) : 0u;
  for (int size = 2; size <= n2; size <<= 1) {
    for (int stride = size >> 1; stride >= 128; stride >>= 1) {
      __syncthreads();
      if (i0 < n2) *reinterpret_cast<uint4*>(sk + i0) = make_uint4(k[0], k[1], k[2], k[3]);
      __syncthreads();
      if (i0 < n2) {
        const uint4 o = *reinterpret_cast<const uint4*>(sk + (i0 ^ stride));
        const bool want_max = ((i0 & size) == 0) == ((i0 & stride) == 0);
        k[0] = want_max ? max(k[0], o.x) : min(k[0], o.x); k[1] = want_max ? max(k[1], o.y) : min(k[1], o.y);
        k[2] = want_max ? max(k[2], o.z) : min(k[2], o.z); k[3] = want_max ? max(k[3], o.w) : min(k[3], o.w);
      }
    }
    for (int stride = min(size >> 1, 64); stride >= 4; stride >>= 1) {
      const bool want_max = ((i0 & size) == 0) == ((i0 & stride) == 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, k[j], stride >> 2);
        k[j] = want_max ? max(k[j], o) : min(k[j], o);
      }
    }
    auto order = [&](uint32_t& a, uint32_t& b, int i) { const uint32_t hi = max(a, b), lo = min(a, b); const bool d = (i & size) == 0; a = d ? hi : lo; b = d ? lo : hi; };
    if (size >= 4) { order(k[0], k[2], i0); order(k[1], k[3], i0 + 1); }
    order(k[0], k[1], i0);
    order(k[2], k[3], i0 + 2);
  }
  __syncthreads();
  if (i0 < n2) *reinterpret_cast<uint4*>(sk + i0) = make_uint4(k[0], k[1], k[2], k[3]);
  __syncthreads();
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

// Nucleus, min-p and the draw over a list that holds every element that can be kept: n of them, in index order, of which
// those from `x_thr` on passed top-k.  z: the sum of exponentials, or 0 to sum the list.  First CTA only.
__device__ void finish_in_list(Row& r, int n, const uint32_t* sk, float x_thr, float mx, float z, bool nucleus, float tp, float mp,
                               float u, int* out) {
  const float* lx = r.bins;
  const int* li = reinterpret_cast<const int*>(r.bins + kCap);
  auto e_of = [&](float x) { return x >= x_thr ? __expf(x - mx) : 0.f; };
  constexpr int kPer = kCap / kThreads;
  float e[kPer], local = 0.f;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = r.tid * kPer + j;
    e[j] = i < n ? e_of(lx[i]) : 0.f;
    local += e[j];
  }
  if (z == 0.f) block_excl(r, local, &z);
  float e_cut = fmaxf(mp, FLT_MIN);            // the largest probability is exp(0) / Z
  if (nucleus) e_cut = fmaxf(e_cut, e_of(key_value(sk[first_reaching(r, sk, n, 0.f, tp * z, e_of)])));
  local = 0.f;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    e[j] = e[j] >= e_cut ? e[j] : 0.f;
    local += e[j];
  }
  float total;
  const float lo = block_excl(r, local, &total);
  const float target = u * total;
  // the first kept index whose running sum passes the target; rounding at the end: the last kept index
  if (r.tid == 0) { r.sh->bc_i = INT_MAX; r.sh->last = -1; }
  __syncthreads();
  float acc = lo;
  int last = -1;
  bool hit = false;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (e[j] > 0.f) {
      last = r.tid * kPer + j;
      acc += e[j];
      if (!hit && target < acc) { hit = true; atomicMin(&r.sh->bc_i, last); }
    }
  }
  if (last >= 0) atomicMax(&r.sh->last, last);
  __syncthreads();
  if (r.tid == 0) {
    const int at = r.sh->bc_i != INT_MAX ? r.sh->bc_i : r.sh->last;
    *out = at >= 0 ? li[at] : -1;
  }
}

__global__ void __launch_bounds__(kThreads)
sample_kernel(int* out, const float* logits, int ld, int V, int slice, int in_smem, int greedy_alone, const float* temperature, const int* top_k,
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
  const int seg = ((r.n + kWarps - 1) / kWarps + 127) & ~127;
  r.seg0 = min(r.n, r.warp * seg);
  r.seg1 = min(r.n, r.seg0 + seg);
  const float* lg = logits + static_cast<size_t>(row) * ld + r.base;
  r.lg = lg;
  const bool quads = (reinterpret_cast<uintptr_t>(lg) & 15) == 0;      // the row's start decides: ld need not be a multiple of 4
  const float T = temperature ? temperature[row] : 1.0f;
  if (T <= 0.f) {
    if (greedy_alone) {
      // The CTAs do not fit the chip at once: a greedy row, which reads its logits once, gives its cluster's places back (128 rows x
      // 128256, all greedy: 36 us, 44 with the whole cluster at work; 64 rows 26 either way.  Where all are resident the cluster is
      // the faster one: one row of 128256 13 us).
      if (r.rank) return;
      r.n = V; r.nc = 1;
    }
    // arg-max, lowest index on ties: a thread sees its indices in ascending order, then packed (ordered value, ~index)
    uint32_t bk = 0, bi = 0;
    bool any = false;
    auto see = [&](float v, int i) { const uint32_t kx = ordered_key(v); if (!any || kx > bk) { bk = kx; bi = i; any = true; } };
    const int nq = quads ? r.n / 4 : 0;
    int i = r.tid;
    for (; i + 7 * kThreads < nq; i += 8 * kThreads) {
      float4 v[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = reinterpret_cast<const float4*>(lg)[i + t * kThreads];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int at = 4 * (i + t * kThreads);
        see(v[t].x, at); see(v[t].y, at + 1); see(v[t].z, at + 2); see(v[t].w, at + 3);
      }
    }
    for (; i < nq; i += kThreads) {
      const float4 v = reinterpret_cast<const float4*>(lg)[i];
      see(v.x, 4 * i); see(v.y, 4 * i + 1); see(v.z, 4 * i + 2); see(v.w, 4 * i + 3);
    }
#pragma unroll 8
    for (i = 4 * nq + r.tid; i < r.n; i += kThreads) see(lg[i], i);
    unsigned long long best = any ? (static_cast<unsigned long long>(bk) << 32) | (0xFFFFFFFFu - (r.base + bi)) : 0ull;
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
    r.sync();
    if (r.rank == 0 && r.tid == 0) {
      for (int q = 1; q < r.nc; ++q) {
        const unsigned long long t = *r.cl().map_shared_rank(bw, q);
        best = t > best ? t : best;
      }
      out[row] = static_cast<int>(0xFFFFFFFFu - static_cast<uint32_t>(best & 0xFFFFFFFFu));
    }
    r.sync();        // the other CTAs' words stay readable until here
    return;
  }
  const float invT = r.invT = 1.0f / fmaxf(T, 1e-6f);
  float mx = -INFINITY;
  {
    const int nq = quads && r.in_smem ? r.n / 4 : 0;
#pragma unroll 8
    for (int i = r.tid; i < nq; i += kThreads) {
      float4 v = reinterpret_cast<const float4*>(lg)[i];
      v.x *= invT; v.y *= invT; v.z *= invT; v.w *= invT;
      reinterpret_cast<float4*>(r.xs)[i] = v;
      mx = max_nan(max_nan(mx, v.x, v.y), v.z, v.w);
    }
#pragma unroll 8
    for (int i = 4 * nq + r.tid; i < r.n; i += kThreads) {
      const float v = lg[i] * invT;
      if (r.in_smem) r.xs[i] = v;
      mx = max_nan(mx, v);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max_nan(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (r.lane == 0) sh.part[r.ex][r.warp].f = mx;
  {
    const int buf = r.exchange();
    mx = -INFINITY;
    for (int q = 0; q < r.nc; ++q) mx = max_nan(mx, r.lane < kWarps ? r.peer(q)->part[buf][r.lane].f : -INFINITY);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max_nan(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (mx != mx) {
    if (r.rank == 0 && r.tid == 0) out[row] = -1;
    r.sync();      // other CTAs may still read this one's maximum
    return;
  }
  const float u = u_in ? u_in[row] : hash_uniform(seed ? seed[row] : 0ull, step);
  const float tp = top_p ? top_p[row] : 1.0f;
  const bool nucleus = tp < 1.0f && tp > 0.f;      // a target of zero keeps everything
  const float mp = min_p ? min_p[row] : 0.f;
  float x_thr = -INFINITY;                         // the k-th largest scaled logit
  const int k = top_k ? top_k[row] : 0;
  if (k > 0 && k < V) {
    Interval iv = Interval::whole(mx);
    float above = 0.f, own = 0.f;
    const float kf = static_cast<float>(k);
    auto one = [](float) { return 1.0f; };
    iv.enter(min(find_bin(r, iv, kf, false, above, own, one).bin, kBins - 1));
    while (own > 0.f && !iv.single() && (k <= kCap ? above + own > kCap : own > kCap))
      iv.enter(min(find_bin(r, iv, kf, false, above, own, one).bin, kBins - 1));
    if (k <= kCap && above + own <= kCap) {
      // every candidate fits the list: the first CTA finishes the row there
      const int n = gather(r, [&](float x) { return iv.reached(x); });
      r.sync();
      if (r.rank == 0) {
        const uint32_t* sk = sorted_list(r, min(n, kCap));
        finish_in_list(r, min(n, kCap), sk, key_value(sk[min(k, n) - 1]), mx, 0.f, nucleus, tp, mp, u, out + row);
      }
      return;           // nobody reads another CTA's memory after the barrier above
    }
    if (iv.single()) {
      x_thr = key_value(iv.klo);
    } else {
      const int n = min(kCap, gather(r, [&](float x) { return iv.inside(x); }));
      r.sync();
      if (r.rank == 0) {
        const int at = min(n - 1, max(0, k - static_cast<int>(above) - 1));
        const uint32_t* sk = sorted_list(r, n);
        if (r.tid == 0) sh.bc_f = n > 0 ? key_value(sk[at]) : -INFINITY;
      }
      r.sync();
      x_thr = r.peer(0)->bc_f;
      r.sync();
    }
  }
  // exponentials stand for the probabilities throughout: a cut on p = e / Z is a cut on e, the draw compares with u times
  // the sum of what is kept
  auto e_of = [&](float x) -> float { return x >= x_thr ? __expf(x - mx) : 0.f; };
  float e_cut = fmaxf(mp, FLT_MIN);                // the largest probability is exp(0) / Z
  if (nucleus) {
    // smallest set of the largest probabilities whose mass reaches top_p of the total
    Interval iv = Interval::whole(mx);
    float above = 0.f, own = 0.f;
    Cut c = find_bin(r, iv, tp, true, above, own, e_of);
    const float target = tp * c.all;
    if (c.bin < kBins) {
      iv.enter(c.bin);
      int n;
      if (c.few <= kCap) {
        n = gather(r, [&](float x) { return iv.reached(x); });
        if (n <= kCap) {
          // a peaked row: everything that can be kept fits the list
          r.sync();
          if (r.rank == 0) finish_in_list(r, n, sorted_list(r, n), x_thr, mx, c.all, true, tp, mp, u, out + row);
          return;
        }
      }
      // a unit-wide bin holds at least its mass over its largest element: skip a gather that cannot fit
      bool deeper = own > __expf(-static_cast<float>(c.bin)) * kCap;
      while (!iv.single()) {
        if (!deeper) {
          n = gather(r, [&](float x) { return iv.inside(x); });
          if (n <= kCap) break;
        }
        deeper = false;
        iv.enter(min(find_bin(r, iv, target, false, above, own, e_of).bin, kBins - 1));
      }
      float cut;
      if (iv.single()) {
        cut = e_of(key_value(iv.klo));
      } else {
        r.sync();
        if (r.rank == 0) {
          const uint32_t* sk = sorted_list(r, n);
          const int pos = n > 0 ? first_reaching(r, sk, n, above, target, e_of) : 0;
          if (r.tid == 0) sh.bc_f = n > 0 ? e_of(key_value(sk[pos])) : 0.f;
        }
        r.sync();
        cut = r.peer(0)->bc_f;
        r.sync();
      }
      e_cut = fmaxf(e_cut, cut);
    }
  }
  auto p_of = [&](float x) -> float {
    const float e = e_of(x);
    return e >= e_cut ? e : 0.f;
  };
  // inverse CDF in index order: sums of the warps' contiguous parts, then the warp whose part holds the target walks it
  float ps = 0.f;
  r.each_of_part([&](float x) { ps += p_of(x); });
  ps = warp_sum(ps);
  if (r.lane == 0) sh.part[r.ex][r.warp].f = ps;
  const int buf = r.exchange();
  // lane l holds the four parts 4l .. 4l + 3 in vocabulary order
  constexpr int kPer = kMaxCluster * kWarps / 32;
  float w4[kPer], mine = 0.f;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int g = r.lane * kPer + j;
    w4[j] = g < r.nc * kWarps ? r.peer(g / kWarps)->part[buf][g % kWarps].f : 0.f;
    mine += w4[j];
  }
  const float incl = warp_incl(mine, r.lane);
  const float target = u * __shfl_sync(0xffffffffu, incl, 31);
  float acc = incl - mine, lo_at = 0.f, lo_last = 0.f;
  int at = INT_MAX, last = -1;      // part that holds the target; last part that keeps anything
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (w4[j] > 0.f) {
      last = r.lane * kPer + j; lo_last = acc;
      if (at == INT_MAX && target < acc + w4[j]) { at = last; lo_at = acc; }
      acc += w4[j];
    }
  }
  const int part_at = __reduce_min_sync(0xffffffffu, at), part_last = __reduce_max_sync(0xffffffffu, last);
  const int part = part_at != INT_MAX ? part_at : part_last;
  const float lo = __shfl_sync(0xffffffffu, part_at != INT_MAX ? lo_at : lo_last, max(part, 0) / kPer);
  if (part < 0) {
    if (r.rank == 0 && r.tid == 0) out[row] = -1;
  } else if (part == r.rank * kWarps + r.warp) {
    float run = lo;
    int pick = -1, kept = -1, have;
    // eight 128-element steps at a time, their scans side by side; only the step that is hit is looked into
    for (int i0 = r.seg0; i0 < r.seg1 && pick < 0; i0 += 128 * 8) {
      float sums[8], scan[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float4 v = r.quad(i0 + t * 128 + 4 * r.lane, &have);
        sums[t] = p_of(v.x) + p_of(v.y) + p_of(v.z) + p_of(v.w);     // a missing element is NaN, which is kept by no cut
        scan[t] = sums[t];
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const float w = __shfl_up_sync(0xffffffffu, scan[t], o);
          if (r.lane >= o) scan[t] += w;
        }
      int step_hit = -1, step_kept = -1;      // step * 32 + lane
      float lo_hit = 0.f, lo_kept = 0.f;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const uint32_t any = __ballot_sync(0xffffffffu, sums[t] > 0.f);
        const uint32_t hit = __ballot_sync(0xffffffffu, sums[t] > 0.f && target < run + scan[t]);
        const float below = run + (scan[t] - sums[t]);
        if (any) { const int l = 31 - __clz(any); step_kept = t * 32 + l; lo_kept = __shfl_sync(0xffffffffu, below, l); }
        if (hit && step_hit < 0) { const int l = __ffs(hit) - 1; step_hit = t * 32 + l; lo_hit = __shfl_sync(0xffffffffu, below, l); }
        run += __shfl_sync(0xffffffffu, scan[t], 31);
      }
      const int sl = step_hit >= 0 ? step_hit : step_kept;
      if (sl >= 0) {
        // the four elements of the lane that holds the target, or of the last lane that keeps anything
        const int i = i0 + (sl >> 5) * 128 + 4 * (sl & 31);
        const float4 v = r.quad(i, &have);
        const float q4[4] = {p_of(v.x), p_of(v.y), p_of(v.z), p_of(v.w)};
        float a = step_hit >= 0 ? lo_hit : lo_kept;
        bool done = false;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (q4[j] > 0.f && !done) { kept = i + j; a += q4[j]; done = step_hit >= 0 && target < a; }
        if (step_hit >= 0) pick = kept;
      }
    }
    if (pick < 0) pick = kept;     // rounding left the target at or past the part's end: its last kept index
    if (r.lane == 0) out[row] = pick >= 0 ? r.base + pick : -1;
  }
  r.sync();                     // other CTAs may still read this one's sums
}

}  // namespace

extern "C" {

// logits f32 [rows][ld]; temperature / top_p / min_p f32 [rows] and top_k int32 [rows] (each may be NULL =
// neutral); u f32 [rows] uniform variates in [0,1) or NULL to hash (seed[row], step); out int32 [rows].
int plow_sample(int* out, const float* logits, int ld, int rows, int V, const float* temperature, const int* top_k,
                const float* top_p, const float* min_p, const float* u, const void* seed, uint64_t step, void* stream) {
  if (rows <= 0 || V <= 0) return -1;
  const int room = 2 * plow::sm_count();
  // CTAs per row: as many as it takes for the slices to fit two CTAs to an SM, and beyond that up to eight while all CTAs are resident
  // at once (64 rows x 8192, no filter: 15.7 us as 256 CTAs, 28.1 as 512) and a slice has 2048 elements (32 rows x 8192, no filter:
  // 14.3 us as slices of 2048, 17.6 of 1024).
  int nc = 1;
  while (nc < kMaxCluster && (V + nc - 1) / nc > kSlice) nc <<= 1;
  while (nc < kMaxCluster && static_cast<long long>(rows) * 2 * nc <= room && V / (2 * nc) >= 2048) nc <<= 1;
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
  cudaError_t e = cudaLaunchKernelEx(&cfg, sample_kernel, out, logits, ld, V, slice, in_smem, static_cast<int>(static_cast<long long>(rows) * nc > room), temperature, top_k, top_p, min_p, u,
                                     static_cast<const unsigned long long*>(seed), static_cast<unsigned long long>(step));
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

}  // extern "C"
