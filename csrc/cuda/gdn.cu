// Gated delta-rule linear attention: causal depthwise conv + SiLU, gates, state recurrence and the gated
// output norm.  Semantics (runtime/nvidia/op_qwen_gdn.cuh:1237-1247, runtime/common/dev_isa.h:1259-1280):
//   x      = SiLU(conv1d_causal(qkv, width W))               per channel, history [W-1] kept per sequence
//   q, k   = x_q / sqrt(|x_q|^2 + 1e-6), x_k / sqrt(|x_k|^2 + 1e-6)       per key head (128 dims)
//   alpha  = exp(-exp(A_log) * softplus(a + dt_bias)),  beta = bf16(sigmoid(b))
//   S     <- alpha S;   S <- S + beta (v - S k) (x) k;   o = S q / sqrt(d)       S[V][K] f32 per (sequence, v head)
//   out    = RMSNorm(o) * gamma * SiLU(z)                                  per (token, v head)
//
// A call is two kernels.  gdn_prep_kernel does what is independent per token: convolution, SiLU, the norms, the gates and
// the dot products of neighbouring tokens, into f32 scratch, and lists the runs (consecutive rows of one sequence).
// gdn_recur_kernel walks the runs.  Row i of S depends on the whole of k but on no other row, so a (run, v head) is cut
// into four items of 32 rows and one prompt fills 128 SMs with hv = 32; inside a CTA eight lanes share a pair of rows
// (16 of the 128 columns each, in registers), so a dot product is three shuffles deep.  Two tokens are taken per step:
//     p1 = S k1, p2 = S k2, r1 = S q1, r2 = S q2               against the same S, one round of shuffles for all four
//     d1 = b1 (v1 - a1 p1),  d2 = b2 (v2 - a2 (a1 p2 + d1 k1.k2))
//     o1 = a1 r1 + d1 k1.q1,  o2 = a2 (a1 r2 + d1 k1.q2) + d2 k2.q2,   S <- a1 a2 S + a2 d1 k1 + d2 k2
// which is the recurrence above with its sums regrouped, all in f32.  What bounds it is the serial chain of a step (packed
// FMAs of the four products, the shuffles, the two updates), about 330 clocks for two tokens; the inputs of the next tokens
// come in by cp.async meanwhile.  One CTA per (run, head) that also convolved, with 128 columns per thread and two block
// reductions per token, took 5180 us for 2048 tokens and 32 heads (2.5 us a token, and each CTA counted its run's rows one
// load after another).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"

namespace {

constexpr int kD = 128;          // head dim
constexpr int kW = 4;            // convolution width

__device__ __forceinline__ float silu(float x) { return x / (1.0f + __expf(-x)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// f32 scratch of a call, in this order: [rows][hk][k 128 | q 128], [rows][hv][v 128], [rows][hk] dots (k.q, kp.k, kp.q, 0)
// with kp the key of the row before in the same run, [rows][hv] gates (alpha, beta); then int2 runs[rows] (first row, rows)
// and the number of runs.
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
    gates = reinterpret_cast<float2*>(dots + rows * hk);
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

// One warp per (row block, head slot): slots [0, hk) are the q and k channels of a key head, [hk, hk + hv) the v channels
// of a v head; a lane owns four consecutive channels.  The last block column lists the runs.
__global__ void __launch_bounds__(256)
gdn_prep_kernel(float* scratch, const float* conv_state, const __nv_bfloat16* qkvz, int ld_qkvz, const __nv_bfloat16* ba, int ld_ba,
                const float* conv_w, const float* a_log, const float* dt_bias, const int* pos, const int* seq, int rows,
                int hk, int hv, int row_block, int vec) {
  plow::pdl_launch_dependents();
  plow::pdl_wait();
  const Scratch sc(scratch, rows, hk, hv);
  if (blockIdx.x == gridDim.x - 1) {
    if (blockIdx.y == 0) list_runs(sc.runs, pos, seq, rows);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int slot = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (slot >= hk + hv) return;
  const bool is_v = slot >= hk;
  const int vh = slot - hk;
  const int C = (2 * hk + hv) * kD;
  const int ch0 = (is_v ? 2 * hk * kD + vh * kD : slot * kD) + lane * 4;       // first channel; k's follow hk * 128 later
  const int n_ch = is_v ? 1 : 2;
  float w[2][4][kW];
  for (int g = 0; g < n_ch; ++g)
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int j = 0; j < kW; ++j) w[g][c][j] = conv_w[static_cast<size_t>(ch0 + g * hk * kD + c) * kW + j];
  const int ra = blockIdx.x * row_block, rb = min(rows, ra + row_block);
  // the row before the block is convolved too where the first row continues it: its key enters the dots
  const int r_first = !is_v && ra > 0 && continues(pos, seq, ra) ? ra - 1 : ra;
  float kp[4] = {0.f, 0.f, 0.f, 0.f};
  for (int r = r_first; r < rb; ++r) {
    if (pos[r] < 0) continue;
    int back = 0;                                   // rows of the same run before this one, up to W - 1
    while (back < kW - 1 && continues(pos, seq, r - back)) ++back;
    const bool cont = back > 0;
    const bool fresh = pos[r] - back == 0;          // the run starts its sequence (only asked where back < W - 1)
    const float* cs = conv_state + static_cast<size_t>(seq[r]) * C * (kW - 1);
    float y[2][4];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (g >= n_ch) break;
      const int ch = ch0 + g * hk * kD;
      float x[kW][4];                               // oldest first; the newest is this row
#pragma unroll
      for (int j = 0; j < kW; ++j) {
        const int age = kW - 1 - j;
        if (age <= back) {
          const __nv_bfloat16* src = qkvz + static_cast<size_t>(r - age) * ld_qkvz + ch;
          if (vec) {
            const uint2 u = *reinterpret_cast<const uint2*>(src);
            const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&u.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
            x[j][0] = __bfloat162float(lo.x); x[j][1] = __bfloat162float(lo.y);
            x[j][2] = __bfloat162float(hi.x); x[j][3] = __bfloat162float(hi.y);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) x[j][c] = __bfloat162float(src[c]);
          }
        } else {
          // history holds the W - 1 inputs before the run, oldest first
#pragma unroll
          for (int c = 0; c < 4; ++c) x[j][c] = fresh ? 0.f : cs[static_cast<size_t>(ch + c) * (kW - 1) + back + j];
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float a = w[g][c][kW - 1] * x[kW - 1][c];
#pragma unroll
        for (int j = 0; j < kW - 1; ++j) a = fmaf(w[g][c][j], x[j][c], a);
        y[g][c] = silu(a);
      }
    }
    if (is_v) {
      *reinterpret_cast<float4*>(sc.v + (static_cast<size_t>(r) * hv + vh) * kD + lane * 4) = make_float4(y[0][0], y[0][1], y[0][2], y[0][3]);
      if (lane == 0) {
        const float bb = __bfloat162float(ba[static_cast<size_t>(r) * ld_ba + vh]);
        const float aa = __bfloat162float(ba[static_cast<size_t>(r) * ld_ba + hv + vh]) + dt_bias[vh];
        const float sp = aa > 20.f ? aa : log1pf(__expf(aa));
        const float alpha = __expf(-__expf(a_log[vh]) * sp);
        const float beta = __bfloat162float(__float2bfloat16(1.0f / (1.0f + __expf(-bb))));
        sc.gates[static_cast<size_t>(r) * hv + vh] = make_float2(alpha, beta);
      }
      continue;
    }
    float qq = 0.f, kk = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) { qq = fmaf(y[0][c], y[0][c], qq); kk = fmaf(y[1][c], y[1][c], kk); }
    qq = warp_sum(qq); kk = warp_sum(kk);
    const float iq = rsqrtf(qq + 1e-6f), ik = rsqrtf(kk + 1e-6f);
    float dkq = 0.f, dpk = 0.f, dpq = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      y[0][c] *= iq; y[1][c] *= ik;
      dkq = fmaf(y[1][c], y[0][c], dkq);
      dpk = fmaf(kp[c], y[1][c], dpk);
      dpq = fmaf(kp[c], y[0][c], dpq);
    }
    dkq = warp_sum(dkq); dpk = warp_sum(dpk); dpq = warp_sum(dpq);
    if (r >= ra) {
      float* dst = sc.kq + (static_cast<size_t>(r) * hk + slot) * 2 * kD + lane * 4;
      *reinterpret_cast<float4*>(dst) = make_float4(y[1][0], y[1][1], y[1][2], y[1][3]);
      *reinterpret_cast<float4*>(dst + kD) = make_float4(y[0][0], y[0][1], y[0][2], y[0][3]);
      // the products with the row before are used only where it belongs to the same run
      if (lane == 0) sc.dots[static_cast<size_t>(r) * hk + slot] = make_float4(dkq, cont ? dpk : 0.f, cont ? dpq : 0.f, 0.f);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) kp[c] = y[1][c];
  }
}

constexpr int kRowsItem = 32;                   // state rows of an item
constexpr int kSplit = kD / kRowsItem;
constexpr int kRecurThreads = 128;              // 16 row pairs x 8 lanes
constexpr int kTok = 8;                         // tokens per stage
constexpr int kStagesR = 3;
constexpr int kConvItem = 1024;                 // channels per item of the history update
struct __align__(16) Stage {
  float kq[kTok][2 * kD];
  float v[kTok][kRowsItem];
  float4 dots[kTok];
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

// Items: (run, v head, quarter of the state rows), then (run, 1024 channels) for the convolution history.
__global__ void __launch_bounds__(kRecurThreads)
gdn_recur_kernel(__nv_bfloat16* out, float* conv_state, float* ssm_state, const float* scratch, const __nv_bfloat16* qkvz, int ld_qkvz,
                 const int* pos, const int* seq, int rows, int hk, int hv, int vec) {
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
    const int kh = h / (hv / hk);
    const int pair = tid >> 3, l8 = tid & 7;
    const int v0 = quarter * kRowsItem;            // first state row of the item
    float* Sg = ssm_state + ((static_cast<size_t>(seq[r0]) * hv + h) * kD + v0 + 2 * pair) * kD + 4 * l8;
    const int n_st = (n + kTok - 1) / kTok;
    auto load_stage = [&](int i) {
      Stage& s = st[i % kStagesR];
      const int t0 = i * kTok, nt = min(kTok, n - t0);
      const size_t r = static_cast<size_t>(r0 + t0);
      for (int e = tid; e < nt * (2 * kD / 4); e += kRecurThreads) {
        const int t = e / (2 * kD / 4), c = e % (2 * kD / 4);
        cp_async16(&s.kq[t][4 * c], sc.kq + ((r + t) * hk + kh) * 2 * kD + 4 * c);
      }
      if (tid < nt * (kRowsItem / 4)) {
        const int t = tid / (kRowsItem / 4), c = tid % (kRowsItem / 4);
        cp_async16(&s.v[t][4 * c], sc.v + ((r + t) * hv + h) * kD + v0 + 4 * c);
      }
      if (tid >= 64 && tid < 64 + nt) cp_async16(&s.dots[tid - 64], sc.dots + (r + tid - 64) * hk + kh);
      if (tid >= 96 && tid < 96 + nt) cp_async8(&s.gates[tid - 96], sc.gates + (r + tid - 96) * hv + h);
    };
    __syncthreads();                               // the stages of the previous item are read
#pragma unroll
    for (int i = 0; i < kStagesR - 1; ++i) {
      if (i < n_st) load_stage(i);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // two state rows, columns {32 j + 4 l8 .. + 3}
    f32x2 S[2][8];
    if (pos[r0] == 0) {
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int j = 0; j < 8; ++j) S[a][j] = 0ull;
    } else {
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float* g = Sg + a * kD + 32 * j;
          const float4 f = vec ? *reinterpret_cast<const float4*>(g) : make_float4(g[0], g[1], g[2], g[3]);
          S[a][2 * j] = pack2(f.x, f.y);
          S[a][2 * j + 1] = pack2(f.z, f.w);
        }
    }
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
        const float4 dt1 = s.dots[t];
        const float* kq1 = s.kq[t] + 4 * l8;
        f32x2 k1[8], q1[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(kq1 + 32 * j), b = *reinterpret_cast<const ulonglong2*>(kq1 + kD + 32 * j);
          k1[2 * j] = a.x; k1[2 * j + 1] = a.y; q1[2 * j] = b.x; q1[2 * j + 1] = b.y;
        }
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
        const float4 dt2 = s.dots[t + 1];
        const float* kq2 = s.kq[t + 1] + 4 * l8;
        f32x2 k2[8], q2[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(kq2 + 32 * j), b = *reinterpret_cast<const ulonglong2*>(kq2 + kD + 32 * j);
          k2[2 * j] = a.x; k2[2 * j + 1] = a.y; q2[2 * j] = b.x; q2[2 * j + 1] = b.y;
        }
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
          const float s2 = g1.x * p2[a] + d1[a] * dt2.y;                    // S after token 1, times k2
          d2[a] = g2.y * ((a ? vv2.y : vv2.x) - g2.x * s2);
          const float e1 = g2.x * d1[a];
          const f32x2 c1 = pack2(e1, e1), c2 = pack2(d2[a], d2[a]);
#pragma unroll
          for (int j = 0; j < 8; ++j) S[a][j] = fma2(c2, k2[j], fma2(c1, k1[j], mul2(al, S[a][j])));
        }
        const float dd1 = up ? d1[1] : d1[0], dd2 = up ? d2[1] : d2[0];
        const float o = (l8 & 1) ? g2.x * (g1.x * ro + dd1 * dt2.z) + dd2 * dt2.x : g1.x * ro + dd1 * dt1.x;
        if (l8 < 4) op[static_cast<size_t>(i * kTok + t + (l8 & 1)) * hv * kD + (up ? 1 : 0)] = __float2bfloat16(o * scale);
      }
    }
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
  return static_cast<int64_t>(rows) * (4ll * (hk * 2 * kD + hv * kD + 4 * hk + 2 * hv) + 8) + 16;
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
  const int vec = ((reinterpret_cast<uintptr_t>(qkvz) & 7) == 0 && ld_qkvz % 4 == 0) ? 1 : 0;
  // rows per warp of the first kernel: one while the rows leave SMs idle, eight beyond (a block convolves one row twice)
  const int row_block = rows <= 256 ? 1 : 8;
  plow::launch_serial(gdn_prep_kernel, dim3((rows + row_block - 1) / row_block + 1, (hk + hv + 7) / 8), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
      scratch, conv_state, static_cast<const __nv_bfloat16*>(qkvz), ld_qkvz, static_cast<const __nv_bfloat16*>(ba), ld_ba, conv_w, a_log, dt_bias,
      pos, seq, rows, hk, hv, row_block, vec);
  const long long most = static_cast<long long>(rows) * (hv * kSplit + ((2 * hk + hv) * kD + kConvItem - 1) / kConvItem);
  const int grid = static_cast<int>(most < 148 * 4 ? most : 148 * 4);
  plow::launch_serial(gdn_recur_kernel, dim3(grid), dim3(kRecurThreads), 0, reinterpret_cast<cudaStream_t>(stream),
      static_cast<__nv_bfloat16*>(out), conv_state, ssm_state, static_cast<const float*>(scratch), static_cast<const __nv_bfloat16*>(qkvz), ld_qkvz,
      pos, seq, rows, hk, hv, (reinterpret_cast<uintptr_t>(ssm_state) & 15) == 0 ? 1 : 0);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 4000 + static_cast<int>(e);
}

int plow_gated_norm(void* out, const void* o, const void* z, int ld_z, int z_ofs, const float* gamma, int rows, int heads,
                    int hd, float eps, void* stream) {
  if (rows <= 0) return -1;
  const long long items = static_cast<long long>(rows) * heads;
  plow::launch_serial(gated_norm_kernel, dim3(static_cast<unsigned>((items + 7) / 8)), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), 
      static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(z), ld_z, z_ofs,
      gamma, rows, heads, hd, eps);
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
