// Gated delta-rule linear attention: causal depthwise conv + SiLU, gates, state recurrence and the gated
// output norm.  Semantics (runtime/nvidia/op_qwen_gdn.cuh:1237-1247, runtime/common/dev_isa.h:1259-1280):
//   x      = SiLU(conv1d_causal(qkv, width W))               per channel, history [W-1] kept per sequence
//   q, k   = x_q / sqrt(|x_q|^2 + 1e-6), x_k / sqrt(|x_k|^2 + 1e-6)       per key head (128 dims)
//   alpha  = exp(-exp(A_log) * softplus(a + dt_bias)),  beta = bf16(sigmoid(b))
//   S     <- alpha S;   S <- S + beta (v - S k) (x) k;   o = S q / sqrt(d)       S[V][K] f32 per (sequence, v head)
//   out    = RMSNorm(o) * gamma * SiLU(z)                                  per (token, v head)
//
// A call is two kernels, above kShortRows rows three.  gdn_prep_kernel does what is independent per token: convolution, SiLU,
// the norms, the gates and the dot products of neighbouring tokens, into f32 scratch, and lists the runs (consecutive rows of one sequence).  The
// recurrence walks the runs: gdn_long_kernel those of kLongRun rows and more, gdn_short_kernel the others (decode; up to
// kShortRows rows take it alone).  Row i of S depends on the whole of k but on no other row, so a (run, v head) is cut into
// four items of 32 rows and one prompt fills 128 SMs with hv = 32; inside a CTA eight lanes share a pair of rows (16 of the
// 128 columns each, in registers), so a dot product is three shuffles deep.  Several tokens (4 or 2) are taken per step:
// with c_i = a_1 .. a_i,  P_i = S k_i and R_i = S q_i all against the S before the step (one round of shuffles for all),
//     s_i = c_i P_i + sum_{j<i} (a_{j+1} .. a_i) d_j (k_j . k_i),   d_i = b_i (v_i - s_i)
//     o_i = c_i R_i + sum_{j<=i} (a_{j+1} .. a_i) d_j (k_j . q_i),  S  <- c_n S + sum_j (a_{j+1} .. a_n) d_j k_j
// which is the recurrence above with its sums regrouped, all in f32.  What bounds it is the issue of the packed FMAs and
// the shared-memory reads of k and q (every thread reads its 16 columns), and between them the serial part of a step: one
// warp per scheduler, 565 instructions and 1780 clocks for four tokens (issue slots 33 % busy, the stalls are fixed latencies).  2048 tokens of one prompt, 32 heads: 530 us, of
// which 460 the recurrence (two tokens a step: 725) and 55 the preparation; 64 decode rows 67 us.  One CTA per (run, head)
// that also convolved, with 128 columns per thread and two block reductions a token, took 4880 us and 191 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "tmap.cuh"

namespace {

constexpr int kD = 128;          // head dim
constexpr int kW = 4;            // convolution width

__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// f32 scratch of a call, in this order: [rows][hk][k 128 | q 128], [rows][hv][v 128], [rows][hk][2 x 4] dots: k_{r-d}.q_r for
// d = 0 .. 3, then k_{r-d}.k_r for d = 1 .. 3 (zero where row r - d is of another run), [rows][hv] gates (alpha, beta), runs.
struct Scratch {
  float* kq;
  float* v;
  float4* dots;
  float2* gates;
  int* runs;       // first row of run i at [i], one past its last row at [rows + i], number of runs at [2 rows]
  __host__ __device__ Scratch(float* base, size_t rows, int hk, int hv) {
    kq = base;
    v = kq + rows * hk * 2 * kD;
    dots = reinterpret_cast<float4*>(v + rows * hv * kD);
    gates = reinterpret_cast<float2*>(dots + 2 * rows * hk);
    runs = reinterpret_cast<int*>(gates + rows * hv);
  }
};

// row r continues the run of row r - 1
__device__ __forceinline__ bool continues(const int* pos, const int* seq, int r) {
  return r > 0 && pos[r] >= 0 && pos[r - 1] >= 0 && seq[r - 1] == seq[r] && pos[r - 1] + 1 == pos[r];
}

// The runs of the call in row order, by one block: starts and ends are compacted separately and pair up by index.
__device__ void list_runs(int* runs, const int* pos, const int* seq, int rows) {
  __shared__ int cnt[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int base_s = 0, base_e = 0;
  for (int r0 = 0; r0 < rows; r0 += blockDim.x) {
    const int r = r0 + threadIdx.x;
    const bool live = r < rows && pos[r] >= 0;
    const bool start = live && !continues(pos, seq, r);
    const bool end = live && (r + 1 >= rows || !continues(pos, seq, r + 1));
    const uint32_t ms = __ballot_sync(0xffffffffu, start), me = __ballot_sync(0xffffffffu, end);
    __syncthreads();
    if (lane == 0) { cnt[0][warp] = __popc(ms); cnt[1][warp] = __popc(me); }
    __syncthreads();
    int os = base_s, oe = base_e;
    for (int w = 0; w < nw; ++w) {
      if (w < warp) { os += cnt[0][w]; oe += cnt[1][w]; }
      base_s += cnt[0][w]; base_e += cnt[1][w];
    }
    const uint32_t below = (1u << lane) - 1;
    if (start) runs[os + __popc(ms & below)] = r;
    if (end) runs[rows + oe + __popc(me & below)] = r + 1;
  }
  if (threadIdx.x == 0) runs[2 * rows] = base_s;
}

__device__ __forceinline__ void unpack4(uint2 u, float* x) {
  const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&u.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  x[0] = __bfloat162float(lo.x); x[1] = __bfloat162float(lo.y); x[2] = __bfloat162float(hi.x); x[3] = __bfloat162float(hi.y);
}

// One warp per (RB rows, head slot): slots [0, hk) are the q and k channels of a key head, [hk, hk + hv) the v channels of a
// v head; a lane owns four consecutive channels and keeps its taps and the last three keys in registers while it walks the
// rows, the next row's inputs already requested.  What bounds it is instruction issue (about 300 per row of a key head, slots 53 % busy with the 15
// warps an SM that 126 registers leave), so
// the walk is a loop: unrolled over its rows, with every row's inputs up front, it took 80 us for 2048 rows and spent a
// quarter of the time fetching instructions.  The first block column lists the runs.
template <int RB>
__global__ void __launch_bounds__(256)
gdn_prep_kernel(float* scratch, const float* conv_state, const __nv_bfloat16* qkvz, int ld_qkvz, const __nv_bfloat16* ba, int ld_ba,
                const float* conv_w, const float* a_log, const float* dt_bias, const int* pos, const int* seq, int rows,
                int hk, int hv, int vec) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const Scratch sc(scratch, rows, hk, hv);
  if (blockIdx.x == 0) {
    if (blockIdx.y == 0) list_runs(sc.runs, pos, seq, rows);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int slot = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (slot >= hk + hv) return;
  const bool is_v = slot >= hk;
  const int vh = slot - hk;
  const int C = (2 * hk + hv) * kD;
  const int ra = (blockIdx.x - 1) * RB, rb = min(rows, ra + RB);
  // lane i: row ra - 6 + i (three rows before the block whose keys enter the dots, three more that those convolve).  How
  // many rows before it are of its run, counted up to lane 0
  constexpr int kBefore = 2 * (kW - 1);
  static_assert(kBefore + RB <= 32, "one lane per row");
  const int rl = ra - kBefore + lane;
  const bool there = rl >= 0 && rl < rb;
  const int pl = there ? pos[rl] : -1, sl = there ? seq[rl] : 0;
  const int pp = __shfl_up_sync(0xffffffffu, pl, 1), ps = __shfl_up_sync(0xffffffffu, sl, 1);
  const uint32_t joins = __ballot_sync(0xffffffffu, lane > 0 && pl >= 0 && pp >= 0 && sl == ps && pp + 1 == pl);
  // consecutive set bits of `joins` ending at this lane's bit
  const int bl = __clz(~(joins << (31 - lane)));
  // first lane (row) to walk: the block's own rows, for keys up to three rows of the run before it
  const int reach = min(kW - 1, __shfl_sync(0xffffffffu, bl, kBefore));
  const int i0 = is_v ? kBefore : kBefore - reach;
  struct Chan { float w[4][kW]; float x[kW][4]; uint2 next; int ch; };
  auto load_row = [&](int i, int ch) -> uint2 {
    const int r = ra - kBefore + i;
    if (r < 0 || r >= rb) return make_uint2(0u, 0u);
    const __nv_bfloat16* src = qkvz + static_cast<size_t>(r) * ld_qkvz + ch;
    if (vec & 1) return *reinterpret_cast<const uint2*>(src);
    const uint16_t* h = reinterpret_cast<const uint16_t*>(src);
    return make_uint2(h[0] | (static_cast<uint32_t>(h[1]) << 16), h[2] | (static_cast<uint32_t>(h[3]) << 16));
  };
  auto begin = [&](Chan& c, int ch) {
    c.ch = ch;
    uint2 raw[kW - 1];
#pragma unroll
    for (int j = 0; j < kW - 1; ++j) raw[j] = load_row(i0 - (kW - 1) + j, ch);
    c.next = load_row(i0, ch);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float* w = conv_w + static_cast<size_t>(ch + k) * kW;
      const float4 f = vec & 2 ? *reinterpret_cast<const float4*>(w) : make_float4(w[0], w[1], w[2], w[3]);
      c.w[k][0] = f.x; c.w[k][1] = f.y; c.w[k][2] = f.z; c.w[k][3] = f.w;
    }
#pragma unroll
    for (int j = 0; j < kW - 1; ++j) unpack4(raw[j], c.x[j + 1]);
  };
  // SiLU(convolution) of row i, whose run holds `back` rows before it
  auto conv_row = [&](Chan& c, int i, int back, int p, int s, float* y) {
#pragma unroll
    for (int j = 0; j < kW - 1; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) c.x[j][k] = c.x[j + 1][k];
    unpack4(c.next, c.x[kW - 1]);
    c.next = load_row(i + 1, c.ch);
    if (p < 0) return;
    if (back < kW - 1) {
      // inputs before the run: history holds its W - 1 last ones, oldest first; a sequence that starts here has none
      float hist[4 * (kW - 1)];                    // [channel][age]
      const float* cs = conv_state + (static_cast<size_t>(s) * C + c.ch) * (kW - 1);
#pragma unroll
      for (int u = 0; u < kW - 1; ++u) {
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p != back) f = vec & 4 ? reinterpret_cast<const float4*>(cs)[u] : make_float4(cs[4 * u], cs[4 * u + 1], cs[4 * u + 2], cs[4 * u + 3]);
        hist[4 * u] = f.x; hist[4 * u + 1] = f.y; hist[4 * u + 2] = f.z; hist[4 * u + 3] = f.w;
      }
      // tap j lies back + j places into the history
#pragma unroll
      for (int b = 0; b < kW - 1; ++b)
        if (back == b) {
#pragma unroll
          for (int j = 0; j + b < kW - 1; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) c.x[j][k] = hist[k * (kW - 1) + b + j];
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float a = c.w[k][kW - 1] * c.x[kW - 1][k];
#pragma unroll
      for (int j = 0; j < kW - 1; ++j) a = fmaf(c.w[k][j], c.x[j][k], a);
      y[k] = silu(a);
    }
  };
  if (is_v) {
    Chan cv;
    begin(cv, 2 * hk * kD + vh * kD + lane * 4);
#pragma unroll 1
    for (int i = kBefore; i < kBefore + RB; ++i) {
      const int r = ra - kBefore + i;
      const int p = __shfl_sync(0xffffffffu, pl, i), s = __shfl_sync(0xffffffffu, sl, i), back = __shfl_sync(0xffffffffu, bl, i);
      float y[4];
      conv_row(cv, i, back, p, s, y);
      if (p >= 0)
        *reinterpret_cast<float4*>(sc.v + (static_cast<size_t>(r) * hv + vh) * kD + lane * 4) = make_float4(y[0], y[1], y[2], y[3]);
    }
    // gates: lane i takes row ra + i
    const int r = ra + lane;
    if (lane < RB && r < rb && pos[r] >= 0) {
      const float bb = __bfloat162float(ba[static_cast<size_t>(r) * ld_ba + vh]);
      const float aa = __bfloat162float(ba[static_cast<size_t>(r) * ld_ba + hv + vh]) + dt_bias[vh];
      const float sp = aa > 20.f ? aa : log1pf(__expf(aa));
      const float alpha = __expf(-__expf(a_log[vh]) * sp);
      const float beta = __bfloat162float(__float2bfloat16(1.0f / (1.0f + __expf(-bb))));
      sc.gates[static_cast<size_t>(r) * hv + vh] = make_float2(alpha, beta);
    }
    return;
  }
  Chan cq, ck;
  begin(cq, slot * kD + lane * 4);
  begin(ck, hk * kD + slot * kD + lane * 4);
  float kh[kW][4];                     // normalised keys of this row and the three before it (index: distance)
#pragma unroll
  for (int d = 0; d < kW; ++d)
#pragma unroll
    for (int c = 0; c < 4; ++c) kh[d][c] = 0.f;
#pragma unroll 1
  for (int i = i0; i < kBefore + RB; ++i) {
    const int r = ra - kBefore + i;
    const int p = __shfl_sync(0xffffffffu, pl, i), s = __shfl_sync(0xffffffffu, sl, i), back = __shfl_sync(0xffffffffu, bl, i);
#pragma unroll
    for (int d = kW - 1; d > 0; --d)
#pragma unroll
      for (int c = 0; c < 4; ++c) kh[d][c] = kh[d - 1][c];
    float y[4];
    conv_row(ck, i, back, p, s, kh[0]);
    conv_row(cq, i, back, i < kBefore ? -1 : p, s, y);       // a row before the block only moves the taps on
    if (p < 0) continue;
    float kk = 0.f, qq = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) kk = fmaf(kh[0][c], kh[0][c], kk);
    const float ik = rsqrtf(warp_sum(kk) + 1e-6f);
#pragma unroll
    for (int c = 0; c < 4; ++c) kh[0][c] *= ik;
    if (i < kBefore) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) qq = fmaf(y[c], y[c], qq);
    const float iq = rsqrtf(warp_sum(qq) + 1e-6f);
    float dot[8];
#pragma unroll
    for (int d = 0; d < 8; ++d) dot[d] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      y[c] *= iq;
#pragma unroll
      for (int d = 0; d < kW; ++d) dot[d] = fmaf(kh[d][c], y[c], dot[d]);
#pragma unroll
      for (int d = 1; d < kW; ++d) dot[3 + d] = fmaf(kh[d][c], kh[0][c], dot[3 + d]);
    }
    // eight sums over 32 lanes: halve the values three times (lane bits 0 .. 2 then name the value), finish over the rest
#pragma unroll
    for (int o = 1, n = 4; o <= 4; o <<= 1, n >>= 1) {
      const bool hi = lane & o;
#pragma unroll
      for (int d = 0; d < n; ++d) {
        const float keep = hi ? dot[d + n] : dot[d], give = hi ? dot[d] : dot[d + n];
        dot[d] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], 8);
    dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], 16);
    // lane bit 0 chose the upper four, bit 1 the upper two of those, bit 2 the upper one
    const int idx = ((lane & 1) << 2) | (lane & 2) | ((lane >> 2) & 1);
    const int dist = idx < 4 ? idx : idx - 3;
    float* dst = sc.kq + (static_cast<size_t>(r) * hk + slot) * 2 * kD + lane * 4;
    *reinterpret_cast<float4*>(dst) = make_float4(kh[0][0], kh[0][1], kh[0][2], kh[0][3]);
    *reinterpret_cast<float4*>(dst + kD) = make_float4(y[0], y[1], y[2], y[3]);
    if (lane < 8) reinterpret_cast<float*>(sc.dots + (static_cast<size_t>(r) * hk + slot) * 2)[idx] = idx < 7 && dist <= back ? dot[0] : 0.f;
  }
}

constexpr int kRowsItem = 32;                   // state rows of an item
constexpr int kSplit = kD / kRowsItem;
constexpr int kRecurThreads = 128;              // 16 row pairs x 8 lanes
constexpr int kTok = 8;                         // tokens per stage
constexpr int kStagesR = 3;
constexpr int kConvItem = kRecurThreads;        // channels per item of the history update: one per thread
constexpr int kLongRun = 4;                     // rows from which a run is walked four tokens at a time
constexpr int kShortRows = 64;                  // rows up to which a call is a decode step (or as short as one)
struct __align__(16) Stage {
  float kq[kTok][2 * kD];
  float v[kTok][kRowsItem];
  float4 dots[kTok][2];
  float2 gates[kTok];
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 unpack2(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

// Tokens [t0, t0 + nt) of a run into a stage; the other tokens of the stage are made neutral (no decay, no update).
__device__ __forceinline__ void load_tokens(Stage& s, const Scratch& sc, size_t r, int nt, int hk, int hv, int kh, int h, int v0) {
  const int tid = threadIdx.x % kRecurThreads;
#pragma unroll
  for (int u = 0; u < kTok * 2 * kD / 4 / kRecurThreads; ++u) {
    const int e = tid + u * kRecurThreads, t = e / (2 * kD / 4), c = e % (2 * kD / 4);
    if (t < nt) cp_async16(&s.kq[t][4 * c], sc.kq + ((r + t) * hk + kh) * 2 * kD + 4 * c);
    else *reinterpret_cast<float4*>(&s.kq[t][4 * c]) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tid < 64) {
    const int t = tid / (kRowsItem / 4), c = tid % (kRowsItem / 4);
    if (t < nt) cp_async16(&s.v[t][4 * c], sc.v + ((r + t) * hv + h) * kD + v0 + 4 * c);
    else *reinterpret_cast<float4*>(&s.v[t][4 * c]) = make_float4(0.f, 0.f, 0.f, 0.f);
  } else if (tid < 64 + 2 * kTok) {
    const int t = (tid - 64) >> 1, c = tid & 1;
    if (t < nt) cp_async16(&s.dots[t][c], sc.dots + ((r + t) * hk + kh) * 2 + c);
    else s.dots[t][c] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else if (tid >= 96 && tid < 96 + kTok) {
    const int t = tid - 96;
    if (t < nt) cp_async8(&s.gates[t], sc.gates + (r + t) * hv + h);
    else s.gates[t] = make_float2(1.f, 0.f);
  }
}

// two state rows, columns {32 j + 4 l8 .. + 3} of each
__device__ __forceinline__ void load_state(f32x2 S[2][8], const float* Sg, bool fresh, int vec) {
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float* g = Sg + a * kD + 32 * j;
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!fresh) f = vec ? *reinterpret_cast<const float4*>(g) : make_float4(g[0], g[1], g[2], g[3]);
      S[a][2 * j] = pack2(f.x, f.y);
      S[a][2 * j + 1] = pack2(f.z, f.w);
    }
}
__device__ __forceinline__ void store_state(const f32x2 S[2][8], float* Sg, int vec) {
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 lo = unpack2(S[a][2 * j]), hi = unpack2(S[a][2 * j + 1]);
      float* g = Sg + a * kD + 32 * j;
      if (vec) *reinterpret_cast<float4*>(g) = make_float4(lo.x, lo.y, hi.x, hi.y);
      else { g[0] = lo.x; g[1] = lo.y; g[2] = hi.x; g[3] = hi.y; }
    }
}
__device__ __forceinline__ void load_cols(f32x2* k, const float* src) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(src + 32 * j);
    k[2 * j] = a.x; k[2 * j + 1] = a.y;
  }
}

// Runs of kLongRun rows and more, four tokens a step.  Items: (run, v head, quarter of the state rows).  One block per SM
// of two independent halves, each with an item and a barrier of its own: the first 148 items then lie on different SMs
// (single-item blocks were placed two to an SM while a third of the SMs stayed idle).
constexpr int kHalves = 2;
__global__ void __launch_bounds__(kHalves * kRecurThreads)
gdn_long_kernel(__nv_bfloat16* out, float* ssm_state, const float* scratch, const int* pos, const int* seq, int rows, int hk, int hv,
                int vec) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  extern __shared__ __align__(16) uint8_t long_smem[];
  const int half = threadIdx.x / kRecurThreads;
  Stage* st = reinterpret_cast<Stage*>(long_smem) + half * kStagesR;
  auto sync_half = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "n"(kRecurThreads) : "memory"); };
  const Scratch sc(const_cast<float*>(scratch), rows, hk, hv);
  const int tid = threadIdx.x % kRecurThreads;
  const int per_run = hv * kSplit, n_items = sc.runs[2 * rows] * per_run;
  const int pair = tid >> 3, l8 = tid & 7;
  const float scale = rsqrtf(static_cast<float>(kD));
  for (int item = half * gridDim.x + blockIdx.x; item < n_items; item += kHalves * gridDim.x) {
    const int run = item / per_run, h = (item % per_run) / kSplit, quarter = item % kSplit;
    const int r0 = sc.runs[run], n = sc.runs[rows + run] - r0;
    if (n < kLongRun) continue;
    const int kh = h / (hv / hk);
    const int v0 = quarter * kRowsItem;            // first state row of the item
    float* Sg = ssm_state + ((static_cast<size_t>(seq[r0]) * hv + h) * kD + v0 + 2 * pair) * kD + 4 * l8;
    const int n_st = (n + kTok - 1) / kTok, n_blk = (n + 3) / 4;
    sync_half();                               // the stages of the previous item are read
#pragma unroll
    for (int i = 0; i < kStagesR - 1; ++i) {
      if (i < n_st) load_tokens(st[i], sc, static_cast<size_t>(r0) + i * kTok, min(kTok, n - i * kTok), hk, hv, kh, h, v0);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    f32x2 S[2][8];
    load_state(S, Sg, pos[r0] == 0, vec);
    __nv_bfloat16* op = out + static_cast<size_t>(r0) * hv * kD + h * kD + v0 + 2 * pair;
    // stage i becomes readable; stage i + kStagesR - 1 is requested into the place of stage i - 1, which all threads left
    auto advance = [&](int i) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStagesR - 2) : "memory");
      sync_half();
      const int nx = i + kStagesR - 1;
      if (nx < n_st) load_tokens(st[nx % kStagesR], sc, static_cast<size_t>(r0) + nx * kTok, min(kTok, n - nx * kTok), hk, hv, kh, h, v0);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    advance(0);
    f32x2 q[4][8];
#pragma unroll
    for (int t = 0; t < 4; ++t) load_cols(q[t], st[0].kq[t] + kD + 4 * l8);
    for (int b = 0; b < n_blk; ++b) {
      const Stage& s = st[(b >> 1) % kStagesR];
      const int t0 = (b & 1) * 4;
      f32x2 k[4][8];
#pragma unroll
      for (int t = 0; t < 4; ++t) load_cols(k[t], s.kq[t0 + t] + 4 * l8);
      float al[4], be[4], vv[2][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 g = s.gates[t0 + t];
        al[t] = g.x; be[t] = g.y;
        const float2 v2 = *reinterpret_cast<const float2*>(&s.v[t0 + t][2 * pair]);
        vv[0][t] = v2.x; vv[1][t] = v2.y;
      }
      // key-key products of the step: kk1[t] = k_{t-1}.k_t and so on
      const float4 e1 = s.dots[t0 + 1][1], e2 = s.dots[t0 + 2][1], e3 = s.dots[t0 + 3][1];
      const int my_t = l8 & 3, my_a = l8 >> 2;                // the output this lane finishes
      const float4 kq = s.dots[t0 + my_t][0];
      float R[2][4], P[2][4];
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[t] = fma2(S[a][j], q[t][j], acc[t]);
#pragma unroll
        for (int t = 0; t < 4; ++t) { const float2 f = unpack2(acc[t]); R[a][t] = f.x + f.y; }
      }
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[t] = fma2(S[a][j], k[t][j], acc[t]);
#pragma unroll
        for (int t = 0; t < 4; ++t) { const float2 f = unpack2(acc[t]); P[a][t] = f.x + f.y; }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int t = 0; t < 4; ++t) P[a][t] += __shfl_xor_sync(0xffffffffu, P[a][t], o);
      // R: eight values over eight lanes, one left per lane (row l8 >> 2, token l8 & 3)
      float ro;
      {
        float x[4];
        const bool b2 = l8 & 4, b1 = l8 & 2, b0 = l8 & 1;
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = (b2 ? R[1][t] : R[0][t]) + __shfl_xor_sync(0xffffffffu, b2 ? R[0][t] : R[1][t], 4);
        const float y0 = (b1 ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, b1 ? x[0] : x[2], 2);
        const float y1 = (b1 ? x[3] : x[1]) + __shfl_xor_sync(0xffffffffu, b1 ? x[1] : x[3], 2);
        ro = (b0 ? y1 : y0) + __shfl_xor_sync(0xffffffffu, b0 ? y0 : y1, 1);
      }
      // the queries of the next step, while the serial part runs
      if (b + 1 < n_blk) {
        if (b & 1) advance((b + 1) >> 1);
        const Stage& sn = st[((b + 1) >> 1) % kStagesR];
        const int tn = ((b + 1) & 1) * 4;
#pragma unroll
        for (int t = 0; t < 4; ++t) load_cols(q[t], sn.kq[tn + t] + kD + 4 * l8);
      }
      // decay products: m_ji = a_{j+1} .. a_i
      const float a12 = al[0] * al[1], a23 = al[1] * al[2], a34 = al[2] * al[3];
      const float a123 = a12 * al[2], a234 = a23 * al[3], a1234 = a12 * a34;
      const f32x2 all = pack2(a1234, a1234);
      float d[2][4];
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        d[a][0] = be[0] * (vv[a][0] - al[0] * P[a][0]);
        d[a][1] = be[1] * (vv[a][1] - (a12 * P[a][1] + al[1] * (d[a][0] * e1.x)));
        d[a][2] = be[2] * (vv[a][2] - (a123 * P[a][2] + a23 * (d[a][0] * e2.y) + al[2] * (d[a][1] * e2.x)));
        d[a][3] = be[3] * (vv[a][3] - (a1234 * P[a][3] + a234 * (d[a][0] * e3.z) + a34 * (d[a][1] * e3.y) + al[3] * (d[a][2] * e3.x)));
        const float c0 = a234 * d[a][0], c1 = a34 * d[a][1], c2 = al[3] * d[a][2];
        const f32x2 w0 = pack2(c0, c0), w1 = pack2(c1, c1), w2 = pack2(c2, c2), w3 = pack2(d[a][3], d[a][3]);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          S[a][j] = fma2(w3, k[3][j], fma2(w2, k[2][j], fma2(w1, k[1][j], fma2(w0, k[0][j], mul2(all, S[a][j])))));
      }
      {
        float dm[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) dm[t] = my_a ? d[1][t] : d[0][t];
        // kq = k_{t-d}.q_t for d = 0 .. 3 of this lane's token
        float o;
        if (my_t == 0) o = al[0] * ro + dm[0] * kq.x;
        else if (my_t == 1) o = a12 * ro + al[1] * (dm[0] * kq.y) + dm[1] * kq.x;
        else if (my_t == 2) o = a123 * ro + a23 * (dm[0] * kq.z) + al[2] * (dm[1] * kq.y) + dm[2] * kq.x;
        else o = a1234 * ro + a234 * (dm[0] * kq.w) + a34 * (dm[1] * kq.z) + al[3] * (dm[2] * kq.y) + dm[3] * kq.x;
        if (4 * b + my_t < n) op[static_cast<size_t>(4 * b + my_t) * hv * kD + my_a] = __float2bfloat16(o * scale);
      }
    }
    store_state(S, Sg, vec);
  }
}

// Runs shorter than kLongRun (every run if `all`), up to two tokens a step.  Items: (run, v head, quarter of the state rows),
// then (run, kConvItem channels) for the convolution history of every run.
__global__ void __launch_bounds__(kRecurThreads)
gdn_short_kernel(__nv_bfloat16* out, float* conv_state, float* ssm_state, const float* scratch, const __nv_bfloat16* qkvz, int ld_qkvz,
                 const int* pos, const int* seq, int rows, int hk, int hv, int vec, int all) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  __shared__ Stage st[kStagesR];
  const Scratch sc(const_cast<float*>(scratch), rows, hk, hv);
  const int tid = threadIdx.x;
  const int C = (2 * hk + hv) * kD;
  const int n_runs = sc.runs[2 * rows];
  const int per_run = hv * kSplit, conv_per = (C + kConvItem - 1) / kConvItem;
  const int n_state = n_runs * per_run, n_items = n_state + n_runs * conv_per;
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    if (item >= n_state) {
      // new history = the last W - 1 inputs of (old history ++ run); the convolution that reads the old one is done
      const int run = (item - n_state) / conv_per, part = (item - n_state) % conv_per;
      const int r0 = sc.runs[run], n = sc.runs[rows + run] - r0;
      const bool fresh = pos[r0] == 0;
      float* cs = conv_state + static_cast<size_t>(seq[r0]) * C * (kW - 1);
      for (int c = part * kConvItem + tid; c < min(C, (part + 1) * kConvItem); c += kRecurThreads) {
        float h[kW - 1];
#pragma unroll
        for (int j = 0; j < kW - 1; ++j) {
          const int back = (kW - 1) - j;            // this slot holds the input `back` steps before the next token
          h[j] = back <= n ? __bfloat162float(qkvz[static_cast<size_t>(r0 + n - back) * ld_qkvz + c])
                           : (fresh ? 0.f : cs[c * (kW - 1) + j + n]);
        }
#pragma unroll
        for (int j = 0; j < kW - 1; ++j) cs[c * (kW - 1) + j] = h[j];
      }
      continue;
    }
    const int run = item / per_run, h = (item % per_run) / kSplit, quarter = item % kSplit;
    const int r0 = sc.runs[run], n = sc.runs[rows + run] - r0;
    if (!all && n >= kLongRun) continue;
    const int kh = h / (hv / hk);
    const int pair = tid >> 3, l8 = tid & 7;
    const int v0 = quarter * kRowsItem;            // first state row of the item
    float* Sg = ssm_state + ((static_cast<size_t>(seq[r0]) * hv + h) * kD + v0 + 2 * pair) * kD + 4 * l8;
    const int n_st = (n + kTok - 1) / kTok;
    auto load_stage = [&](int i) {
      load_tokens(st[i % kStagesR], sc, static_cast<size_t>(r0) + i * kTok, min(kTok, n - i * kTok), hk, hv, kh, h, v0);
    };
    __syncthreads();                               // the stages of the previous item are read
#pragma unroll
    for (int i = 0; i < kStagesR - 1; ++i) {
      if (i < n_st) load_stage(i);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    f32x2 S[2][8];
    load_state(S, Sg, pos[r0] == 0, vec);
    const float scale = rsqrtf(static_cast<float>(kD));
    __nv_bfloat16* op = out + static_cast<size_t>(r0) * hv * kD + h * kD + v0 + 2 * pair;
    for (int i = 0; i < n_st; ++i) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStagesR - 2) : "memory");
      __syncthreads();
      if (i + kStagesR - 1 < n_st) load_stage(i + kStagesR - 1);      // into the stage that was read before the barrier
      asm volatile("cp.async.commit_group;" ::: "memory");
      const Stage& s = st[i % kStagesR];
      const int nt = min(kTok, n - i * kTok);
#pragma unroll 1
      for (int t = 0; t < nt; t += 2) {
        const bool two = t + 1 < nt;
        const float2 g1 = s.gates[t];
        const float2 vv1 = *reinterpret_cast<const float2*>(&s.v[t][2 * pair]);
        const float4 dt1 = s.dots[t][0];
        const float* kq1 = s.kq[t] + 4 * l8;
        f32x2 k1[8], q1[8];
        load_cols(k1, kq1);
        load_cols(q1, kq1 + kD);
        if (!two) {
          f32x2 p[2] = {0ull, 0ull}, q[2] = {0ull, 0ull};
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int a = 0; a < 2; ++a) { p[a] = fma2(S[a][j], k1[j], p[a]); q[a] = fma2(S[a][j], q1[j], q[a]); }
          float ov[2];
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            const float2 pp = unpack2(p[a]), qq = unpack2(q[a]);
            float x = pp.x + pp.y, y = qq.x + qq.y;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) { x += __shfl_xor_sync(0xffffffffu, x, o); y += __shfl_xor_sync(0xffffffffu, y, o); }
            const float d = g1.y * ((a ? vv1.y : vv1.x) - g1.x * x);
            ov[a] = g1.x * y + d * dt1.x;
            const f32x2 al = pack2(g1.x, g1.x), dd = pack2(d, d);
#pragma unroll
            for (int j = 0; j < 8; ++j) S[a][j] = fma2(dd, k1[j], mul2(al, S[a][j]));
          }
          if (l8 < 2) op[static_cast<size_t>(i * kTok + t) * hv * kD + l8] = __float2bfloat16((l8 ? ov[1] : ov[0]) * scale);
          break;
        }
        const float2 g2 = s.gates[t + 1];
        const float2 vv2 = *reinterpret_cast<const float2*>(&s.v[t + 1][2 * pair]);
        const float4 dt2 = s.dots[t + 1][0];
        const float kk2 = s.dots[t + 1][1].x;
        const float* kq2 = s.kq[t + 1] + 4 * l8;
        f32x2 k2[8], q2[8];
        load_cols(k2, kq2);
        load_cols(q2, kq2 + kD);
        f32x2 ap1[2] = {0ull, 0ull}, ap2[2] = {0ull, 0ull}, ar1[2] = {0ull, 0ull}, ar2[2] = {0ull, 0ull};
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            ap1[a] = fma2(S[a][j], k1[j], ap1[a]);
            ap2[a] = fma2(S[a][j], k2[j], ap2[a]);
            ar1[a] = fma2(S[a][j], q1[j], ar1[a]);
            ar2[a] = fma2(S[a][j], q2[j], ar2[a]);
          }
        float p1[2], p2[2], r1[2], r2[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          float2 f = unpack2(ap1[a]); p1[a] = f.x + f.y;
          f = unpack2(ap2[a]); p2[a] = f.x + f.y;
          f = unpack2(ar1[a]); r1[a] = f.x + f.y;
          f = unpack2(ar2[a]); r2[a] = f.x + f.y;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            p1[a] += __shfl_xor_sync(0xffffffffu, p1[a], o);
            p2[a] += __shfl_xor_sync(0xffffffffu, p2[a], o);
          }
        // the outputs are needed by one lane each: token l8 & 1, row (l8 >> 1) & 1 after two exchanges that halve the values
        float rr[2];
        {
          const bool odd = l8 & 1;
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            const float keep = odd ? r2[a] : r1[a], give = odd ? r1[a] : r2[a];
            rr[a] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
          }
        }
        const bool up = l8 & 2;
        float ro = (up ? rr[1] : rr[0]) + __shfl_xor_sync(0xffffffffu, up ? rr[0] : rr[1], 2);
        ro += __shfl_xor_sync(0xffffffffu, ro, 4);
        const float a12 = g1.x * g2.x;
        const f32x2 al = pack2(a12, a12);
        float d1[2], d2[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          d1[a] = g1.y * ((a ? vv1.y : vv1.x) - g1.x * p1[a]);
          const float s2 = g1.x * p2[a] + d1[a] * kk2;                      // S after token 1, times k2
          d2[a] = g2.y * ((a ? vv2.y : vv2.x) - g2.x * s2);
          const float e1 = g2.x * d1[a];
          const f32x2 c1 = pack2(e1, e1), c2 = pack2(d2[a], d2[a]);
#pragma unroll
          for (int j = 0; j < 8; ++j) S[a][j] = fma2(c2, k2[j], fma2(c1, k1[j], mul2(al, S[a][j])));
        }
        const float dd1 = up ? d1[1] : d1[0], dd2 = up ? d2[1] : d2[0];
        const float o = (l8 & 1) ? g2.x * (g1.x * ro + dd1 * dt2.y) + dd2 * dt2.x : g1.x * ro + dd1 * dt1.x;
        if (l8 < 4) op[static_cast<size_t>(i * kTok + t + (l8 & 1)) * hv * kD + (up ? 1 : 0)] = __float2bfloat16(o * scale);
      }
    }
    store_state(S, Sg, vec);
  }
}

// One warp per (row, head): out = RMSNorm(o) * gamma * SiLU(z).
__global__ void gated_norm_kernel(__nv_bfloat16* out, const __nv_bfloat16* o, const __nv_bfloat16* z, int ld_z, int z_ofs,
                                  const float* gamma, int rows, int heads, int hd, float eps) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + wib;
  if (item >= static_cast<long long>(rows) * heads) return;
  const int r = static_cast<int>(item / heads), h = static_cast<int>(item % heads);
  const __nv_bfloat16* src = o + (static_cast<size_t>(r) * heads + h) * hd;
  float ss = 0.f;
  for (int c = lane; c < hd; c += 32) { const float v = __bfloat162float(src[c]); ss += v * v; }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
  const float rs = rsqrtf(ss / hd + eps);
  for (int c = lane; c < hd; c += 32) {
    const float zz = __bfloat162float(z[static_cast<size_t>(r) * ld_z + z_ofs + h * hd + c]);
    out[(static_cast<size_t>(r) * heads + h) * hd + c] = __float2bfloat16(__bfloat162float(src[c]) * rs * gamma[c] * silu(zz));
  }
}

// The same for heads of 128 whose rows are aligned for 8-byte loads: a lane owns four consecutive channels, every load of
// an item is in flight at once (2048 x 32 heads: 31 us with 2-byte loads, the traffic takes 8).
__global__ void __launch_bounds__(256)
gated_norm128_kernel(__nv_bfloat16* out, const __nv_bfloat16* o, const __nv_bfloat16* z, int ld_z, int z_ofs,
                     const float* gamma, int rows, int heads, float eps) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long item = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= static_cast<long long>(rows) * heads) return;
  const int r = static_cast<int>(item / heads), h = static_cast<int>(item % heads);
  const uint2 ou = *reinterpret_cast<const uint2*>(o + item * kD + lane * 4);
  const uint2 zu = *reinterpret_cast<const uint2*>(z + static_cast<size_t>(r) * ld_z + z_ofs + h * kD + lane * 4);
  float x[4], zz[4], g[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) g[c] = gamma[lane * 4 + c];
  unpack4(ou, x);
  unpack4(zu, zz);
  const float ss = warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
  const float rs = rsqrtf(ss / kD + eps);
#pragma unroll
  for (int c = 0; c < 4; ++c) x[c] = x[c] * rs * g[c] * silu(zz[c]);
  const __nv_bfloat162 lo = __floats2bfloat162_rn(x[0], x[1]), hi = __floats2bfloat162_rn(x[2], x[3]);
  *reinterpret_cast<uint2*>(out + item * kD + lane * 4) =
      make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// out = a * sigmoid(gate)   (gated full-attention layers of the hybrid model)
__global__ void sigmoid_gate_kernel(__nv_bfloat16* out, const __nv_bfloat16* a, const __nv_bfloat16* gate, long long n) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16(__bfloat162float(a[i]) / (1.0f + __expf(-__bfloat162float(gate[i]))));
}

}  // namespace

extern "C" {

// Bytes of scratch plow_gdn needs for `rows` rows.
int64_t plow_gdn_scratch_bytes(int rows, int hk, int hv) {
  if (rows <= 0 || hk <= 0 || hv <= 0) return 0;
  return static_cast<int64_t>(rows) * (4ll * (hk * 2 * kD + hv * kD + 8 * hk + 2 * hv) + 8) + 16;
}

// qkvz bf16 [rows][ld_qkvz] = [q (hk*128) | k (hk*128) | v (hv*128) | z ...]; ba bf16 [rows][ld_ba] = [b (hv) | a (hv)];
// conv_w f32 [(2hk+hv)*128][conv]; conv_state f32 [slots][(2hk+hv)*128][conv-1]; ssm_state f32 [slots][hv][128][128];
// out bf16 [rows][hv*128].  A row whose position is 0 starts its sequence from a zero state.  scratch: 16-byte aligned,
// plow_gdn_scratch_bytes.
int plow_gdn(void* out, float* conv_state, float* ssm_state, const void* qkvz, int ld_qkvz, const void* ba, int ld_ba,
             const float* conv_w, const float* a_log, const float* dt_bias, const int* pos, const int* seq, int rows,
             int hk, int hv, int head_dim, int conv, float* scratch, void* stream) {
  if (rows <= 0 || head_dim != kD || conv != kW || hk <= 0 || hv % hk || !scratch) return -1;
  if (reinterpret_cast<uintptr_t>(scratch) & 15) return -3;
  // which inputs of the first kernel are aligned for vector loads: rows, filter taps, history
  const int vec = ((reinterpret_cast<uintptr_t>(qkvz) & 7) == 0 && ld_qkvz % 4 == 0 ? 1 : 0) |
                  ((reinterpret_cast<uintptr_t>(conv_w) & 15) == 0 ? 2 : 0) | ((reinterpret_cast<uintptr_t>(conv_state) & 15) == 0 ? 4 : 0);
  const int vec_s = (reinterpret_cast<uintptr_t>(ssm_state) & 15) == 0 ? 1 : 0;
  cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
  const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(qkvz);
  const __nv_bfloat16* gates = static_cast<const __nv_bfloat16*>(ba);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  // Rows per warp of the first kernel: one while the rows leave SMs idle, eight beyond (a block convolves the keys of three
  // rows before it again).  Up to kShortRows rows the short kernel takes every run: a decode step then is two launches.
  const int units = (hk + hv + 7) / 8;
  if (rows <= 256)
    plow::launch_serial(gdn_prep_kernel<1>, dim3(rows + 1, units), dim3(256), 0, cs, scratch, conv_state, x, ld_qkvz, gates, ld_ba, conv_w,
                        a_log, dt_bias, pos, seq, rows, hk, hv, vec);
  else
    plow::launch_serial(gdn_prep_kernel<8>, dim3((rows + 7) / 8 + 1, units), dim3(256), 0, cs, scratch, conv_state, x, ld_qkvz, gates, ld_ba,
                        conv_w, a_log, dt_bias, pos, seq, rows, hk, hv, vec);
  const float* sc = scratch;
  constexpr int kLongSmem = kHalves * kStagesR * sizeof(Stage);
  static plow::DeviceOnce attr;
  if (rows > kShortRows && plow::ensure_smem(attr, gdn_long_kernel, kLongSmem) != cudaSuccess) return 3000;
  if (rows > kShortRows)
    plow::launch_serial(gdn_long_kernel, dim3(plow::sm_count()), dim3(kHalves * kRecurThreads), kLongSmem, cs, o, ssm_state, sc, pos, seq, rows, hk, hv, vec_s);
  const long long most = static_cast<long long>(rows) * (hv * kSplit + ((2 * hk + hv) * kD + kConvItem - 1) / kConvItem);
  const int room = 4 * plow::sm_count();
  const int grid = static_cast<int>(most < room ? most : room);
  plow::launch_serial(gdn_short_kernel, dim3(grid), dim3(kRecurThreads), 0, cs, o, conv_state, ssm_state, sc, x, ld_qkvz, pos, seq, rows, hk, hv,
                      vec_s, rows > kShortRows ? 0 : 1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

int plow_gated_norm(void* out, const void* o, const void* z, int ld_z, int z_ofs, const float* gamma, int rows, int heads,
                    int hd, float eps, void* stream) {
  if (rows <= 0) return -1;
  const long long items = static_cast<long long>(rows) * heads;
  const bool vec = hd == kD && ld_z % 4 == 0 && z_ofs % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(z)) & 7) == 0;
  if (vec)
    plow::launch_serial(gated_norm128_kernel, dim3(static_cast<unsigned>((items + 7) / 8)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
        static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(z), ld_z, z_ofs, gamma, rows, heads, eps);
  else
    plow::launch_serial(gated_norm_kernel, dim3(static_cast<unsigned>((items + 7) / 8)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
        static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(z), ld_z, z_ofs, gamma, rows, heads, hd, eps);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

int plow_sigmoid_gate(void* out, const void* a, const void* gate, int64_t n, void* stream) {
  if (n <= 0) return -1;
  plow::launch_serial(sigmoid_gate_kernel, dim3(static_cast<unsigned>((n + 255) / 256)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 
      static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(gate), n);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

}  // extern "C"
