// Gated delta rule: a recurrent mixer whose state per (request, head) is a float32 matrix
// S [key channels, value channels], with one decay per (head, key channel).
//
// Per token and head, in this order:
//   S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// so the read-out sees the token's own write. Around it: short causal convolutions with SiLU
// on q, k and v (the last taps - 1 inputs of a request are part of its state), q and k made
// unit vectors per head (q also times dk^-1/2), beta = sigmoid(.), g = exp(-exp(A_log) *
// softplus(low-rank(h) + dt_bias)), and an output stage: o divided by its root mean square
// over the value channels, times a weight, times sigmoid(low-rank gate).
//
// Everything after the projections is float32 in both serving types. A request's state slot
// is one float32 vector: S for every head, stored transposed [heads, dv, dk] so that the key
// channels a lane keeps are contiguous, then the convolution tail [taps - 1, conv channels].
//
// Kernels:
//   delta_prep     one warp per (token, q / k / v head): convolutions, unit vectors; beta, decay, gate
//   delta_conv     one block per request: the convolution tail after this step
//   delta_scan     one block per (request, head, block of value columns): the recurrence over
//                  the request's tokens of this step, from and to the state slot. Columns of S
//                  are independent; a column's dk entries are spread over KS lanes of a warp,
//                  R contiguous ones to a lane, and the two sums over them are shuffles.
//   delta_out      one warp per (token, head): the output stage
// Portions of more than a few tokens run in chunks instead of delta_scan / general_scan (csrc/delta_chunks.cu).
//
// Two forms of the gated rule share these kernels: the decay is one number per (head, key channel)
// from a low-rank pair, or one number per head from a plain projection (`decay_per_head`: the rates
// then hold `heads` columns, which the preparation spreads over the head's channels); the output
// gate is a sigmoid or SiLU (`gate_silu`); the output weight is shared by the heads or has a row
// per head.
//
// The generalized delta rule (general_prep, general_scan) keeps the same state layout. Per token
// and head, with the unit key u = k / sqrt(|k|^2 + 1e-6), a decay w and a removal rate a per
// (head, key channel):
//   S <- diag(w) S - (a * u) (u^T S) + k v^T     (both first terms read the old S);   o = S^T r
// w = exp(-exp(-1/2) * sigmoid(inner + w0)) with `inner` the product of a low-rank pair with tanh
// between its halves, a = sigmoid(proj_a + bias), gate = sigmoid(proj_g).
#include <stdlib.h>

#include "common.cuh"

namespace {

constexpr int MAX_TAPS = 16;
constexpr int SCAN_THREADS = 256; // most threads of a scan block
constexpr int TOKENS = 16;      // tokens staged in shared memory at a time (in each of two buffers)

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(expf(x)); }

struct PrepArgs {
  // the fused projection [tokens, stride]: columns q | k | v | beta
  const void* proj;
  int proj_f32, stride;
  int off_q, off_k, off_v, off_beta;
  // the low-rank pairs' products [tokens, heads dk + heads dv]: decay rates | output gates
  const void* rates;
  int rates_f32;
  int kv_heads, heads, dk, dv, taps;
  const void* conv_w;           // [(2 kv_heads dk + heads dv), taps], the last column is the current token's
  const void* a_log;            // [heads]
  const void* dt_bias;          // [heads dk]
  int w_f32;
  const float* state;           // [slots, state_stride]
  int64_t state_stride, conv_offset;
  const int* request_of;
  const int* cu_q;
  const int* state_slots;
  int num_slots;
  float* q; float* k; float* v; float* beta; float* decay; float* gate;
  unsigned* status;
  int decay_per_head;           // rates: heads decay columns (dt_bias [heads]) instead of heads * dk
  int gate_silu;                // the output gate is z * sigmoid(z) instead of sigmoid(z)
  int w_words;                  // four taps, and conv_w and dt_bias on whole words
};

// One warp per unit of a token: a q head, a k head or a v head. A lane owns the channels lane,
// lane + 32, ... of its unit, convolves them, and for q and k heads the warp sums the squares
// (a lane's chain, then the fixed tree). blockIdx.y walks the units in groups of the block's
// warps; the element-wise outputs (beta, decay, gate) are spread over the same blocks.
constexpr int PREP_MAX_KEY = 256;            // widest q / k head (8 channels per lane)
__global__ void __launch_bounds__(256) delta_prep_kernel(PrepArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int cq = a.kv_heads * a.dk, cv = a.heads * a.dv, cc = 2 * cq + cv;
  const int b = a.request_of[t];
  const int local = t - a.cu_q[b];
  int slot = a.state_slots[b];
  if (slot < 0 || slot >= a.num_slots) {
    if (threadIdx.x == 0 && blockIdx.y == 0) raise_fault(a.status, VOSTI_FAULT_SLOT_RANGE);
    slot = 0;
  }
  const float* tail = a.state + (int64_t)slot * a.state_stride + a.conv_offset;   // [taps - 1, cc]
  const int64_t row = (int64_t)t * a.stride;
  // q | k | v occupy columns off_q .. off_q + cc of the projection in this order
  auto convolved = [&](int c) {
    float acc = 0.f;
    for (int i = 0; i < a.taps; ++i) {
      const int back = a.taps - 1 - i;                  // how many tokens before this one
      float x;
      if (local - back >= 0) x = load_flex(a.proj, a.proj_f32, row - (int64_t)back * a.stride + a.off_q + c);
      else x = tail[(int64_t)(a.taps - 1 + local - back) * cc + c];
      acc = fmaf(load_flex(a.conv_w, a.w_f32, (int64_t)c * a.taps + i), x, acc);
    }
    return acc * sigmoidf_(acc);
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int units = 2 * a.kv_heads + a.heads;
  for (int unit = blockIdx.y * nwarps + warp; unit < units; unit += gridDim.y * nwarps) {
    if (unit < 2 * a.kv_heads) {
      const int c0 = unit * a.dk;                       // q heads, then k heads
      float y[PREP_MAX_KEY / 32];
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < PREP_MAX_KEY / 32; ++j) {
        const int i = lane + 32 * j;
        y[j] = i < a.dk ? convolved(c0 + i) : 0.f;
        ss += y[j] * y[j];
      }
      ss = warp_sum(ss);
      const bool is_q = unit < a.kv_heads;
      const float scale = (1.f / sqrtf(ss + 1e-6f)) * (is_q ? 1.f / sqrtf((float)a.dk) : 1.f);
      float* dst = (is_q ? a.q : a.k) + (int64_t)t * cq + (is_q ? unit : unit - a.kv_heads) * a.dk;
#pragma unroll
      for (int j = 0; j < PREP_MAX_KEY / 32; ++j) {
        const int i = lane + 32 * j;
        if (i < a.dk) dst[i] = y[j] * scale;
      }
    } else {
      const int c0 = (unit - 2 * a.kv_heads) * a.dv;
      for (int i = lane; i < a.dv; i += 32) a.v[(int64_t)t * cv + c0 + i] = convolved(2 * cq + c0 + i);
    }
  }
  const int first = blockIdx.y * blockDim.x + threadIdx.x, step = gridDim.y * blockDim.x;
  for (int h = first; h < a.heads; h += step)
    a.beta[(int64_t)t * a.heads + h] = sigmoidf_(load_flex(a.proj, a.proj_f32, row + a.off_beta + h));
  const int cd = a.heads * a.dk;
  const int rd = a.decay_per_head ? a.heads : cd;           // decay columns of the rates
  const int64_t rrow = (int64_t)t * (rd + cv);
  for (int c = first; c < cd; c += step) {
    const int from = a.decay_per_head ? c / a.dk : c;
    const float rate = load_flex(a.rates, a.rates_f32, rrow + from) + load_flex(a.dt_bias, a.w_f32, from);
    const float speed = expf(load_flex(a.a_log, a.w_f32, c / a.dk));
    a.decay[(int64_t)t * cd + c] = expf(-speed * softplusf_(rate));
  }
  for (int c = first; c < cv; c += step) {
    const float z = load_flex(a.rates, a.rates_f32, rrow + rd + c);
    a.gate[(int64_t)t * cv + c] = a.gate_silu ? z * sigmoidf_(z) : sigmoidf_(z);
  }
}

// The same for heads of 128 channels and up to four taps (WIDE_TAPS): a lane owns four neighbouring channels of its
// unit and a warp takes TOKENS_EACH tokens one after the other, so that the taps' weights, the decay's constants
// and the last inputs stay in registers and a token's inputs and results are whole words; a v head's warp also makes
// its head's beta, decay and gate. The kernel above is bound by its scalar loads (each input read once per tap): 87 us
// for 2,048 tokens of 16 heads (4 key heads); this one was bound by the rounds of loads that a warp waited for (three before its
// first token, 148 registers and so 12 warps an SM: 58 us), so weights come as words, the rows before the first token without
// waiting for its request, and a thread has 72 registers (28 warps an SM; with several tokens a warp 40 to 64 bytes of them lie in local memory): 40 us past the product before it.
constexpr int WIDE_TAPS = 4;

__device__ __forceinline__ void store_four(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ float4 flex_four(const void* p, int is_f32, int64_t i) {       // load_flex of an aligned word
  return is_f32 ? load_four(reinterpret_cast<const float*>(p) + i) : load_four(reinterpret_cast<const bf16*>(p) + i);
}
__device__ __forceinline__ void spread(float4 v, float (&to)[4]) { to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w; }

template <typename T, int TOKENS_EACH>
__global__ void __launch_bounds__(128, 7) delta_prep_wide_kernel(PrepArgs a, int tokens) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int D = 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int units = 2 * a.kv_heads + a.heads;
  const int unit = blockIdx.y * 4 + warp;
  if (unit >= units) return;
  const int cq = a.kv_heads * D, cv = a.heads * D, cc = 2 * cq + cv;
  const int c = unit * D + lane * 4;                       // channel of q | k | v
  const T* const proj = reinterpret_cast<const T*>(a.proj);
  float w[WIDE_TAPS][4], win[WIDE_TAPS][4];                // right-aligned: index WIDE_TAPS - 1 is the current token
#pragma unroll
  for (int k = 0; k < WIDE_TAPS; ++k)
#pragma unroll
    for (int u = 0; u < 4; ++u) win[k][u] = 0.f;
  if (a.w_words) {                                         // four taps: a channel's weights are one word
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 v = flex_four(a.conv_w, a.w_f32, (int64_t)(c + u) * WIDE_TAPS);
      w[0][u] = v.x; w[1][u] = v.y; w[2][u] = v.z; w[3][u] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < WIDE_TAPS; ++k)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int tap = k - (WIDE_TAPS - a.taps);
        w[k][u] = tap >= 0 ? load_flex(a.conv_w, a.w_f32, (int64_t)(c + u) * a.taps + tap) : 0.f;
      }
  }
  const int head = unit - 2 * a.kv_heads;                  // of a v unit
  float speed = 0.f, shift[4] = {0.f, 0.f, 0.f, 0.f};
  if (head >= 0) {
    speed = expf(load_flex(a.a_log, a.w_f32, head));
    if (a.w_words && !a.decay_per_head) {
      spread(flex_four(a.dt_bias, a.w_f32, head * D + lane * 4), shift);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) shift[u] = load_flex(a.dt_bias, a.w_f32, a.decay_per_head ? head : head * D + lane * 4 + u);
    }
  }
  const int rd = a.decay_per_head ? a.heads : a.heads * D;
  const int t_first = blockIdx.x * TOKENS_EACH, t_end = min(tokens, t_first + TOKENS_EACH);
  // a token's words, asked for together
  struct Words { float4 x, gate, rate; };
  auto ask = [&](Words& to, int t) {
    to.x = load_four(proj + (int64_t)t * a.stride + a.off_q + c);
    if (head < 0) return;
    const int64_t row = (int64_t)t * (rd + cv);
    to.gate = flex_four(a.rates, a.rates_f32, row + rd + head * D + lane * 4);
    if (a.decay_per_head) {
      const float r = load_flex(a.rates, a.rates_f32, row + head);
      to.rate = make_float4(r, r, r, r);
    } else {
      to.rate = flex_four(a.rates, a.rates_f32, row + head * D + lane * 4);
    }
  };
  // the rows before the warp's first token, asked for before its request is known (its own from the request's fourth token on)
  float4 before[WIDE_TAPS - 1];
#pragma unroll
  for (int k = 1; k < WIDE_TAPS; ++k) before[k - 1] = load_four(proj + (int64_t)max(t_first - k, 0) * a.stride + a.off_q + c);
  int b = -1, next_first = 0;
#pragma unroll 1
  for (int t = t_first; t < t_end; ++t) {
    Words now = {};
    ask(now, t);
    if (b < 0 || t >= next_first) {                        // a new request (or the warp's first token): fill the window anew
      b = a.request_of[t];
      const int first = a.cu_q[b];
      next_first = a.cu_q[b + 1];
      int slot = a.state_slots[b];
      if (slot < 0 || slot >= a.num_slots) {
        if (lane == 0 && unit == 0) raise_fault(a.status, VOSTI_FAULT_SLOT_RANGE);
        slot = 0;
      }
      const float* const tail = a.state + (int64_t)slot * a.state_stride + a.conv_offset;       // [taps - 1, cc]
      const int local = t - first;
#pragma unroll
      for (int k = 1; k < WIDE_TAPS; ++k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < a.taps) v = k <= local ? (t == t_first ? before[k - 1] : load_four(proj + (int64_t)(t - k) * a.stride + a.off_q + c))
                                       : load_four(tail + (int64_t)(a.taps - 1 + local - k) * cc + c);
        spread(v, win[WIDE_TAPS - 1 - k]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < WIDE_TAPS - 1; ++k)
#pragma unroll
        for (int u = 0; u < 4; ++u) win[k][u] = win[k + 1][u];
    }
    spread(now.x, win[WIDE_TAPS - 1]);
    float y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < WIDE_TAPS; ++k) if (k >= WIDE_TAPS - a.taps) acc = fmaf(w[k][u], win[k][u], acc);
      y[u] = acc * sigmoidf_(acc);
    }
    if (head < 0) {
      const float ss = warp_sum((y[0] * y[0] + y[1] * y[1]) + (y[2] * y[2] + y[3] * y[3]));
      const bool is_q = unit < a.kv_heads;
      const float scale = (1.f / sqrtf(ss + 1e-6f)) * (is_q ? 1.f / sqrtf((float)D) : 1.f);
#pragma unroll
      for (int u = 0; u < 4; ++u) y[u] *= scale;
      store_four((is_q ? a.q : a.k) + (int64_t)t * cq + (is_q ? unit : unit - a.kv_heads) * D + lane * 4, y);
      continue;
    }
    const int64_t at = (int64_t)t * cv + head * D + lane * 4;
    store_four(a.v + at, y);
    float z[4], rate[4];
    spread(now.gate, z);
    spread(now.rate, rate);
#pragma unroll
    for (int u = 0; u < 4; ++u) z[u] = a.gate_silu ? z[u] * sigmoidf_(z[u]) : sigmoidf_(z[u]);
    store_four(a.gate + at, z);
    if (a.decay_per_head) {
      rate[0] = rate[1] = rate[2] = rate[3] = expf(-speed * softplusf_(rate[0] + shift[0]));
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) rate[u] = expf(-speed * softplusf_(rate[u] + shift[u]));
    }
    store_four(a.decay + at, rate);
    if (lane == 0) a.beta[(int64_t)t * a.heads + head] = sigmoidf_(to_f32(proj[(int64_t)t * a.stride + a.off_beta + head]));
  }
}

// The convolution tail of every request after this step: the last taps - 1 rows of
// [old tail ; this step's projection rows]. A thread owns a channel, reads what it needs, then writes.
__global__ void __launch_bounds__(256)
delta_conv_kernel(const void* proj, int proj_f32, int stride, int off_q, int cc, int taps, float* state,
                  int64_t state_stride, int64_t conv_offset, const int* cu_q, const int* state_slots, int num_slots) {
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.x;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= num_slots) return;
  const int start = cu_q[b], n = cu_q[b + 1] - start;
  float* tail = state + (int64_t)slot * state_stride + conv_offset;
  const int keep = taps - 1;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < cc; c += gridDim.y * blockDim.x) {
    float next[MAX_TAPS];
    for (int r = 0; r < keep; ++r) {
      const int idx = n + r;                 // row of [old tail (keep rows) ; projection rows (n)]
      next[r] = idx < keep ? tail[(int64_t)idx * cc + c]
                           : load_flex(proj, proj_f32, (int64_t)(start + idx - keep) * stride + off_q + c);
    }
    for (int r = 0; r < keep; ++r) tail[(int64_t)r * cc + c] = next[r];
  }
}

// KS lanes of a warp share a value column; lane part `ks` keeps key channels ks * R .. ks * R + R - 1
// of it. A warp holds 32 / KS columns, a block (its thread count) / KS. Tokens are staged in
// shared memory TOKENS at a time in two buffers: while one block of tokens is computed, the next
// one's k, q, g, v and beta arrive by cp.async. The staged rows of k, q and g are padded with
// zeros to KS * R channels, so a lane reads its R as 16-byte words. Between two tokens the state
// waits for one chain of multiply-adds and one chain of KS-lane shuffles; both wait on the
// shared-memory and shuffle pipe, so R is chosen for few shuffle steps (see the launcher).
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int KS, int R>
__global__ void __launch_bounds__(SCAN_THREADS)
delta_scan_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                  const float* __restrict__ beta, const float* __restrict__ decay, float* __restrict__ out,
                  float* state, int64_t state_stride, const int* __restrict__ cu_q, const int* __restrict__ state_slots,
                  int num_slots, int kv_heads, int heads, int dk, int dv, int most) {
  extern __shared__ __align__(16) float smem[];
  constexpr int PER_WARP = 32 / KS;             // columns of a warp
  constexpr int PAD = KS * R;                   // staged channels per token
  const int threads = blockDim.x;
  const int COLS = threads / KS;                // value columns of a block (8 or more)
  const int STAGE = TOKENS * (3 * PAD + COLS) + TOKENS;      // floats of one buffer (a multiple of 4)
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * COLS;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= num_slots) return;
  const int start = cu_q[b], n = cu_q[b + 1] - start;
  if (most > 0 && n > most) return;             // a long portion: csrc/delta_chunks.cu
  const int g = h / (heads / kv_heads);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ks = lane / PER_WARP, local = warp * PER_WARP + lane % PER_WARP, col = col0 + local;
  const bool live = col < dv;
  const int r0 = ks * R;
  float* S = state + (int64_t)slot * state_stride + ((int64_t)h * dv + col) * dk;     // this column's dk channels
  float s[R];
  const bool wide = (dk % 4 == 0) && live && r0 + R <= dk;
  if (wide) {
#pragma unroll
    for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(s + i) = *reinterpret_cast<const float4*>(S + r0 + i);
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) s[i] = (live && r0 + i < dk) ? S[r0 + i] : 0.f;
  }
  const int cq = kv_heads * dk, cd = heads * dk, cv = heads * dv;
  // 16-byte copies need every row start on a 16-byte boundary
  const bool vec_k = dk % 4 == 0, vec_v = dv % 4 == 0;
  if (PAD != dk) {                                  // the padding stays zero (lanes beyond dk multiply it with zeros)
    for (int i = threadIdx.x; i < 2 * STAGE; i += threads) smem[i] = 0.f;
    __syncthreads();
  }

  auto stage = [&](int t0, int buf) {
    float* sk = smem + buf * STAGE;
    float* sq = sk + TOKENS * PAD;
    float* sg = sq + TOKENS * PAD;
    float* sv = sg + TOKENS * PAD;
    float* sb = sv + TOKENS * COLS;
    const int count = min(TOKENS, n - t0);
    if (vec_k) {
      const int per = dk / 4;
      for (int i = threadIdx.x; i < count * per; i += threads) {
        const int tt = i / per, c = (i % per) * 4;
        const int64_t t = start + t0 + tt;
        cp_async16(sk + tt * PAD + c, k + t * cq + g * dk + c);
        cp_async16(sq + tt * PAD + c, q + t * cq + g * dk + c);
        cp_async16(sg + tt * PAD + c, decay + t * cd + h * dk + c);
      }
    } else {
      for (int i = threadIdx.x; i < count * dk; i += threads) {
        const int tt = i / dk, c = i % dk;
        const int64_t t = start + t0 + tt;
        cp_async4(sk + tt * PAD + c, k + t * cq + g * dk + c);
        cp_async4(sq + tt * PAD + c, q + t * cq + g * dk + c);
        cp_async4(sg + tt * PAD + c, decay + t * cd + h * dk + c);
      }
    }
    if (vec_v) {
      const int per = COLS / 4;
      for (int i = threadIdx.x; i < count * per; i += threads) {
        const int tt = i / per, c = (i % per) * 4;
        if (col0 + c < dv) cp_async16(sv + tt * COLS + c, v + (int64_t)(start + t0 + tt) * cv + h * dv + col0 + c);
      }
    } else {
      for (int i = threadIdx.x; i < count * COLS; i += threads) {
        const int tt = i / COLS, c = i % COLS;
        if (col0 + c < dv) cp_async4(sv + tt * COLS + c, v + (int64_t)(start + t0 + tt) * cv + h * dv + col0 + c);
      }
    }
    for (int i = threadIdx.x; i < count; i += threads) cp_async4(sb + i, beta + (int64_t)(start + t0 + i) * heads + h);
  };

  float* orow = out + (int64_t)start * cv + h * dv + col;
  if (n > 0) stage(0, 0);
  cp_async_commit();
  for (int t0 = 0, buf = 0; t0 < n; t0 += TOKENS, buf ^= 1) {
    if (t0 + TOKENS < n) stage(t0 + TOKENS, buf ^ 1);         // (its last readers passed the barrier below)
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const float* sk = smem + buf * STAGE + r0;
    const float* sq = sk + TOKENS * PAD;
    const float* sg = sq + TOKENS * PAD;
    const float* sv = smem + buf * STAGE + 3 * TOKENS * PAD + local;
    const float* sb = smem + buf * STAGE + 3 * TOKENS * PAD + TOKENS * COLS;
    const int count = min(TOKENS, n - t0);
    for (int tt = 0; tt < count; ++tt) {
      float kt[R], x[R];
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < R; i += 4) {
        *reinterpret_cast<float4*>(kt + i) = *reinterpret_cast<const float4*>(sk + tt * PAD + i);
        *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(sg + tt * PAD + i);
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        s[i] *= x[i];
        acc[i & 3] = fmaf(s[i], kt[i], acc[i & 3]);
      }
      float dot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
      for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(sq + tt * PAD + i);
#pragma unroll
      for (int o = PER_WARP; o < 32; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      const float u = sb[tt] * (sv[tt * COLS] - dot);
      acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        s[i] = fmaf(kt[i], u, s[i]);
        acc[i & 3] = fmaf(s[i], x[i], acc[i & 3]);
      }
      float read = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
      for (int o = PER_WARP; o < 32; o <<= 1) read += __shfl_xor_sync(0xffffffffu, read, o);
      if (ks == 0 && live) orow[(int64_t)(t0 + tt) * cv] = read;
    }
    __syncthreads();                                         // this buffer may be refilled two rounds on
  }
  cp_async_wait<0>();
  if (wide) {
#pragma unroll
    for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(S + r0 + i) = *reinterpret_cast<const float4*>(s + i);
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (live && r0 + i < dk) S[r0 + i] = s[i];
  }
}

// y[t, h, :] = o / sqrt(mean(o^2) + eps) * w * gate, in the serving type, for the output projection.
template <typename TO>
__global__ void __launch_bounds__(128)
delta_out_kernel(const float* __restrict__ o, const float* __restrict__ gate, const void* __restrict__ w, int w_f32,
                 TO* __restrict__ y, int64_t pairs, int dv, float eps, int heads, int w_per_head) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t pair = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (pair >= pairs) return;
  const float* src = o + pair * dv;
  float ss = 0.f;
  for (int i = lane; i < dv; i += 32) ss += src[i] * src[i];
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / (float)dv + eps);
  const int64_t wbase = w_per_head ? (pair % heads) * dv : 0;
  for (int i = lane; i < dv; i += 32)
    y[pair * dv + i] = from_f32<TO>(src[i] * inv * load_flex(w, w_f32, wbase + i) * gate[pair * dv + i]);
}


// out[t, j] = tanh(x[t, offset + j]) for j < width: the first half of a low-rank pair whose
// halves have a tanh between them, cut out of a wider projection.
template <typename T>
__global__ void __launch_bounds__(256)
tanh_columns_kernel(const T* __restrict__ x, int stride, int offset, int width, T* __restrict__ out, int64_t tokens) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t n = tokens * width;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / width;
    out[i] = from_f32<T>(tanhf(to_f32(x[t * stride + offset + (i - t * width)])));
  }
}

struct GeneralPrepArgs {
  const void* proj;             // [tokens, stride]: columns r | k | v | g | a, each heads * d wide
  int proj_f32, stride;
  int off_r, off_k, off_v, off_g, off_a;
  const float* inner;           // [tokens, heads * d]: the decay's low-rank product
  const void* w0;               // [heads * d]
  const void* a_bias;           // [heads * d]
  int w_f32;
  int heads, d;
  float* r; float* k; float* v; float* decay; float* unit; float* removal; float* gate;
};

// One warp per (token, head): blocks of four warps, blockIdx.y over groups of four heads.
__global__ void __launch_bounds__(128) general_prep_kernel(GeneralPrepArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = (int64_t)t * a.stride;
  const int hd = a.heads * a.d;
  const float rate = 0.6065306597126334f;             // exp(-1/2)
  for (int head = blockIdx.y * 4 + warp; head < a.heads; head += gridDim.y * 4) {
    const int c0 = head * a.d;
    float ss = 0.f;
    for (int i = lane; i < a.d; i += 32) {
      const float x = load_flex(a.proj, a.proj_f32, row + a.off_k + c0 + i);
      ss += x * x;
    }
    ss = warp_sum(ss);
    const float inv = 1.f / sqrtf(ss + 1e-6f);
    for (int i = lane; i < a.d; i += 32) {
      const int c = c0 + i;
      const int64_t o = (int64_t)t * hd + c;
      const float key = load_flex(a.proj, a.proj_f32, row + a.off_k + c);
      const float u = key * inv;
      a.k[o] = key;
      a.unit[o] = u;
      a.removal[o] = sigmoidf_(load_flex(a.proj, a.proj_f32, row + a.off_a + c) + load_flex(a.a_bias, a.w_f32, c)) * u;
      a.r[o] = load_flex(a.proj, a.proj_f32, row + a.off_r + c);
      a.v[o] = load_flex(a.proj, a.proj_f32, row + a.off_v + c);
      a.decay[o] = expf(-rate * sigmoidf_(a.inner[o] + load_flex(a.w0, a.w_f32, c)));
      a.gate[o] = sigmoidf_(load_flex(a.proj, a.proj_f32, row + a.off_g + c));
    }
  }
}

// The same for heads of 128 channels in whole words: a lane owns four neighbouring channels and has its eight
// loads in flight together.
template <typename T>
__global__ void __launch_bounds__(128) general_prep_wide_kernel(GeneralPrepArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int D = 128;
  const int t = blockIdx.x, lane = threadIdx.x & 31, head = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (head >= a.heads) return;
  const T* const row = reinterpret_cast<const T*>(a.proj) + (int64_t)t * a.stride;
  const int c = head * D + lane * 4;
  const int64_t o = (int64_t)t * a.heads * D + c;
  const float rate = 0.6065306597126334f;             // exp(-1/2)
  float key[4], r[4], v[4], z[4], remove[4], inner[4];
  spread(load_four(row + a.off_k + c), key);
  spread(load_four(row + a.off_r + c), r);
  spread(load_four(row + a.off_v + c), v);
  spread(load_four(row + a.off_g + c), z);
  spread(load_four(row + a.off_a + c), remove);
  spread(load_four(a.inner + o), inner);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    remove[u] += load_flex(a.a_bias, a.w_f32, c + u);
    inner[u] += load_flex(a.w0, a.w_f32, c + u);
  }
  store_four(a.k + o, key);
  store_four(a.r + o, r);
  store_four(a.v + o, v);
  const float inv = 1.f / sqrtf(warp_sum((key[0] * key[0] + key[1] * key[1]) + (key[2] * key[2] + key[3] * key[3])) + 1e-6f);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    key[u] *= inv;
    remove[u] = sigmoidf_(remove[u]) * key[u];
    inner[u] = expf(-rate * sigmoidf_(inner[u]));
    z[u] = sigmoidf_(z[u]);
  }
  store_four(a.unit + o, key);
  store_four(a.removal + o, remove);
  store_four(a.decay + o, inner);
  store_four(a.gate + o, z);
}

// The generalized rule's recurrence, laid out as delta_scan: KS lanes share a value column and
// keep R key channels of it each; five vectors of key channels are staged per token (write key,
// read key, decay, unit key, removal = rate * unit key).
template <int KS, int R>
__global__ void __launch_bounds__(SCAN_THREADS)
general_scan_kernel(const float* __restrict__ r, const float* __restrict__ k, const float* __restrict__ v,
                    const float* __restrict__ decay, const float* __restrict__ unit, const float* __restrict__ removal,
                    float* __restrict__ out, float* state, int64_t state_stride, const int* __restrict__ cu_q,
                    const int* __restrict__ state_slots, int num_slots, int heads, int dk, int dv, int most) {
  extern __shared__ __align__(16) float smem[];
  constexpr int PER_WARP = 32 / KS;
  constexpr int PAD = KS * R;
  constexpr int NV = 5;                         // staged vectors of key channels
  const int threads = blockDim.x;
  const int COLS = threads / KS;
  const int STAGE = TOKENS * (NV * PAD + COLS);
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * COLS;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= num_slots) return;
  const int start = cu_q[b], n = cu_q[b + 1] - start;
  if (most > 0 && n > most) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ks = lane / PER_WARP, local = warp * PER_WARP + lane % PER_WARP, col = col0 + local;
  const bool live = col < dv;
  const int r0 = ks * R;
  float* S = state + (int64_t)slot * state_stride + ((int64_t)h * dv + col) * dk;
  float s[R];
  const bool wide = (dk % 4 == 0) && live && r0 + R <= dk;
  if (wide) {
#pragma unroll
    for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(s + i) = *reinterpret_cast<const float4*>(S + r0 + i);
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) s[i] = (live && r0 + i < dk) ? S[r0 + i] : 0.f;
  }
  const int cd = heads * dk, cv = heads * dv;
  const bool vec_k = dk % 4 == 0, vec_v = dv % 4 == 0;
  if (PAD != dk) {
    for (int i = threadIdx.x; i < 2 * STAGE; i += threads) smem[i] = 0.f;
    __syncthreads();
  }
  const float* sources[NV] = {k, r, decay, unit, removal};

  auto stage = [&](int t0, int buf) {
    float* base = smem + buf * STAGE;
    float* sv = base + NV * TOKENS * PAD;
    const int count = min(TOKENS, n - t0);
    if (vec_k) {
      const int per = dk / 4;
      for (int i = threadIdx.x; i < count * per; i += threads) {
        const int tt = i / per, c = (i % per) * 4;
        const int64_t at = (int64_t)(start + t0 + tt) * cd + h * dk + c;
#pragma unroll
        for (int x = 0; x < NV; ++x) cp_async16(base + x * TOKENS * PAD + tt * PAD + c, sources[x] + at);
      }
    } else {
      for (int i = threadIdx.x; i < count * dk; i += threads) {
        const int tt = i / dk, c = i % dk;
        const int64_t at = (int64_t)(start + t0 + tt) * cd + h * dk + c;
#pragma unroll
        for (int x = 0; x < NV; ++x) cp_async4(base + x * TOKENS * PAD + tt * PAD + c, sources[x] + at);
      }
    }
    if (vec_v) {
      const int per = COLS / 4;
      for (int i = threadIdx.x; i < count * per; i += threads) {
        const int tt = i / per, c = (i % per) * 4;
        if (col0 + c < dv) cp_async16(sv + tt * COLS + c, v + (int64_t)(start + t0 + tt) * cv + h * dv + col0 + c);
      }
    } else {
      for (int i = threadIdx.x; i < count * COLS; i += threads) {
        const int tt = i / COLS, c = i % COLS;
        if (col0 + c < dv) cp_async4(sv + tt * COLS + c, v + (int64_t)(start + t0 + tt) * cv + h * dv + col0 + c);
      }
    }
  };

  float* orow = out + (int64_t)start * cv + h * dv + col;
  if (n > 0) stage(0, 0);
  cp_async_commit();
  for (int t0 = 0, buf = 0; t0 < n; t0 += TOKENS, buf ^= 1) {
    if (t0 + TOKENS < n) stage(t0 + TOKENS, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const float* sk = smem + buf * STAGE + r0;
    const float* sr = sk + TOKENS * PAD;
    const float* sw = sr + TOKENS * PAD;
    const float* su = sw + TOKENS * PAD;
    const float* sa = su + TOKENS * PAD;
    const float* sv = smem + buf * STAGE + NV * TOKENS * PAD + local;
    const int count = min(TOKENS, n - t0);
    for (int tt = 0; tt < count; ++tt) {
      float x[R], y[R];
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(su + tt * PAD + i);
#pragma unroll
      for (int i = 0; i < R; ++i) acc[i & 3] = fmaf(s[i], x[i], acc[i & 3]);
      float dot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
      for (int i = 0; i < R; i += 4) {
        *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(sw + tt * PAD + i);
        *reinterpret_cast<float4*>(y + i) = *reinterpret_cast<const float4*>(sa + tt * PAD + i);
      }
#pragma unroll
      for (int o = PER_WARP; o < 32; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      const float value = sv[tt * COLS];
#pragma unroll
      for (int i = 0; i < R; ++i) s[i] = fmaf(-y[i], dot, s[i] * x[i]);
#pragma unroll
      for (int i = 0; i < R; i += 4) {
        *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(sk + tt * PAD + i);
        *reinterpret_cast<float4*>(y + i) = *reinterpret_cast<const float4*>(sr + tt * PAD + i);
      }
      acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        s[i] = fmaf(x[i], value, s[i]);
        acc[i & 3] = fmaf(s[i], y[i], acc[i & 3]);
      }
      float read = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
      for (int o = PER_WARP; o < 32; o <<= 1) read += __shfl_xor_sync(0xffffffffu, read, o);
      if (ks == 0 && live) orow[(int64_t)(t0 + tt) * cv] = read;
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  if (wide) {
#pragma unroll
    for (int i = 0; i < R; i += 4) *reinterpret_cast<float4*>(S + r0 + i) = *reinterpret_cast<const float4*>(s + i);
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (live && r0 + i < dk) S[r0 + i] = s[i];
  }
}

}  // namespace

// Tokens that a warp of the preparation of wide heads takes one after the other (units: heads of q, k and v). A warp waits for each token's
// loads in turn, so one each while the SMs (28 warps of them at a time) run through at most some ten rounds; then four, which
// share the weights and the earlier rows. us, one / four / eight tokens a warp: 24 units, 395 tokens 12.8 / 15.4 / 25.1, 1,000 25.7 /
// 25.5 / 31.1, 1,500 36.0 / 38.2 / 42.8, 2,048 49.0 / 44.0 / 46.6, 3,000 70.6 / 64.6 / 74.0; 48 units, 260 tokens 16.8 / 17.5 / 27.4, 700 34.5 /
// 37.3 / 41.3, 1,000 47.6 / 43.5 / 46.3, 2,048 93.9 / 83.8 / 81.7; 8 units, 2,048 tokens 17.1 / 18.2 / 28.5.
VOSTI_API int vosti_delta_prep_tokens(int tokens, int units) { return (int64_t)tokens * units >= 148 * 270 ? 4 : 1; }

VOSTI_API int vosti_delta_prep(const void* proj, int proj_f32, int stride, int off_q, int off_k, int off_v, int off_beta,
                               const void* rates, int rates_f32, int kv_heads, int heads, int dk, int dv, int taps,
                               const void* conv_w, const void* a_log, const void* dt_bias, int w_f32, float* state,
                               int64_t state_stride, int64_t conv_offset, const int* request_of, const int* cu_q,
                               const int* state_slots, int num_slots, int requests, int tokens, float* q, float* k,
                               float* v, float* beta, float* decay, float* gate, unsigned* status, int decay_per_head,
                               int gate_silu, cudaStream_t stream) {
  VOSTI_REQUIRE(kv_heads > 0 && heads > 0 && heads % kv_heads == 0 && dk > 0 && dv > 0, "delta_prep: bad head sizes");
  VOSTI_REQUIRE(taps >= 1 && taps <= MAX_TAPS, "delta_prep: %d taps (1 to %d are taken)", taps, MAX_TAPS);
  VOSTI_REQUIRE(off_k == off_q + kv_heads * dk && off_v == off_k + kv_heads * dk, "delta_prep: q, k, v must be adjacent columns");
  if (tokens == 0) return VOSTI_OK;
  PrepArgs a = {};
  a.proj = proj; a.proj_f32 = proj_f32; a.stride = stride;
  a.off_q = off_q; a.off_k = off_k; a.off_v = off_v; a.off_beta = off_beta;
  a.rates = rates; a.rates_f32 = rates_f32;
  a.kv_heads = kv_heads; a.heads = heads; a.dk = dk; a.dv = dv; a.taps = taps;
  a.conv_w = conv_w; a.a_log = a_log; a.dt_bias = dt_bias; a.w_f32 = w_f32;
  a.state = state; a.state_stride = state_stride; a.conv_offset = conv_offset;
  a.request_of = request_of; a.cu_q = cu_q; a.state_slots = state_slots; a.num_slots = num_slots;
  a.q = q; a.k = k; a.v = v; a.beta = beta; a.decay = decay; a.gate = gate; a.status = status;
  a.decay_per_head = decay_per_head; a.gate_silu = gate_silu;
  const int cc = 2 * kv_heads * dk + heads * dv;
  VOSTI_REQUIRE(dk <= PREP_MAX_KEY, "delta_prep: %d key channels (at most %d are taken)", dk, PREP_MAX_KEY);
  const int units = 2 * kv_heads + heads;
  const int size = proj_f32 ? 4 : 2, rate_size = rates_f32 ? 4 : 2, rd = decay_per_head ? heads : heads * dk;
  const bool wide = dk == 128 && dv == 128 && taps <= WIDE_TAPS && stride % 4 == 0 && off_q % 4 == 0 && (rd + heads * dv) % 4 == 0 && rd % 4 == 0 &&
                    state_stride % 4 == 0 && conv_offset % 4 == 0 && reinterpret_cast<uintptr_t>(state) % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(proj) % (4 * size) == 0 && reinterpret_cast<uintptr_t>(rates) % (4 * rate_size) == 0 &&
                    ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                      reinterpret_cast<uintptr_t>(decay) | reinterpret_cast<uintptr_t>(gate)) & 15) == 0 && (units + 3) / 4 <= 65535;
  if (wide) {
    a.w_words = taps == WIDE_TAPS && ((reinterpret_cast<uintptr_t>(conv_w) | reinterpret_cast<uintptr_t>(dt_bias)) & (w_f32 ? 15 : 7)) == 0;
    const int each = vosti_delta_prep_tokens(tokens, units);
    const dim3 grid((tokens + each - 1) / each, (units + 3) / 4);
    if (proj_f32) {
      if (each == 4) vosti_launch(delta_prep_wide_kernel<float, 4>, grid, dim3(128), 0, stream, a, tokens);
      else vosti_launch(delta_prep_wide_kernel<float, 1>, grid, dim3(128), 0, stream, a, tokens);
    } else {
      if (each == 4) vosti_launch(delta_prep_wide_kernel<bf16, 4>, grid, dim3(128), 0, stream, a, tokens);
      else vosti_launch(delta_prep_wide_kernel<bf16, 1>, grid, dim3(128), 0, stream, a, tokens);
    }
  } else {
    vosti_launch(delta_prep_kernel, dim3(tokens, (units + 7) / 8 < 65535 ? (units + 7) / 8 : 65535), dim3(256), 0, stream, a);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { vosti_set_error("%s", cudaGetErrorString(e)); return (int)e; }
  // the tail is rewritten only after every token of the step has read the old one
  if (taps > 1)
    vosti_launch(delta_conv_kernel, dim3(requests, (cc + 255) / 256 < 64 ? (cc + 255) / 256 : 64), dim3(256), 0, stream, proj, proj_f32, stride, off_q, cc, taps, state,
                 state_stride, conv_offset, cu_q, state_slots, num_slots);
  VOSTI_LAUNCH_CHECK();
}

// How many key channels a lane keeps (8, 16 or 32). VOSTI_SCAN_ROWS overrides the rule (tuning).
static int scan_rows(int dk) {
  static int forced = -1;
  if (forced < 0) {
    const char* env = getenv("VOSTI_SCAN_ROWS");
    forced = env != nullptr ? atoi(env) : 0;
  }
  if ((forced == 8 || forced == 16 || forced == 32) && dk <= forced * 32 && (forced != 32 || dk <= 256)) return forced;
  return dk <= 32 ? 8 : 16;
}

static int scan_lanes(int dk) {          // of a value column
  int ks = 1;
  while (ks * scan_rows(dk) < dk) ks *= 2;
  return ks;
}

// Value columns of a block of either rule's token-by-token kernel: 8 or more, fewer while the grid would leave SMs idle.
VOSTI_API int vosti_delta_scan_columns(int requests, int heads, int dk, int dv) {
  const int ks = scan_lanes(dk);
  int threads = SCAN_THREADS;
  while (threads > 64 && threads / 2 >= 8 * ks &&
         (int64_t)requests * heads * ((dv + threads / ks - 1) / (threads / ks)) < 296)
    threads /= 2;
  if (threads < 8 * ks) threads = 8 * ks;
  return threads / ks;
}

// `most` > 0: requests that bring more tokens than that are left alone (the chunked kernels take them).
VOSTI_API int vosti_delta_scan(const float* q, const float* k, const float* v, const float* beta, const float* decay,
                               float* out, float* state, int64_t state_stride, const int* cu_q, const int* state_slots,
                               int num_slots, int requests, int kv_heads, int heads, int dk, int dv, int most, cudaStream_t stream) {
  VOSTI_REQUIRE(kv_heads > 0 && heads > 0 && heads % kv_heads == 0 && dk > 0 && dv > 0, "delta_scan: bad head sizes");
  VOSTI_REQUIRE(dk <= 256, "delta_scan: %d key channels (at most 256 are taken)", dk);
  VOSTI_REQUIRE(heads <= 65535, "delta_scan: too many heads");
  VOSTI_REQUIRE(state_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0, "delta_scan: state slots must be 16-byte aligned");
  if (requests == 0) return VOSTI_OK;
  const int rows = scan_rows(dk), ks = scan_lanes(dk), cols = vosti_delta_scan_columns(requests, heads, dk, dv), threads = cols * ks;
  VOSTI_REQUIRE((dv + cols - 1) / cols <= 65535, "delta_scan: too many value channels");
  const dim3 grid(requests, heads, (dv + cols - 1) / cols);
  const size_t smem = 2 * (size_t)(TOKENS * (3 * ks * rows + cols) + TOKENS) * sizeof(float);
#define VOSTI_SCAN(KS, R)                                                                                           \
  do {                                                                                                              \
    static bool configured = false;    /* once per instantiation, to the most a launch of it may ask for */           \
    if (!configured) {                                                                                              \
      cudaFuncSetAttribute(delta_scan_kernel<KS, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,                   \
                           (int)(2 * (size_t)(TOKENS * (3 * KS * R + SCAN_THREADS / KS) + TOKENS) * sizeof(float))); \
      configured = true;                                                                                            \
    }                                                                                                               \
    vosti_launch(delta_scan_kernel<KS, R>, grid, dim3(threads), smem, stream, q, k, v, beta, decay, out, state,    \
                 state_stride, cu_q, state_slots, num_slots, kv_heads, heads, dk, dv, most);                              \
  } while (0)
#define VOSTI_SCAN_KS(R)                                                                                            \
  switch (ks) {                                                                                                     \
    case 1: VOSTI_SCAN(1, R); break;                                                                                \
    case 2: VOSTI_SCAN(2, R); break;                                                                                \
    case 4: VOSTI_SCAN(4, R); break;                                                                                \
    case 8: VOSTI_SCAN(8, R); break;                                                                                \
    case 16: VOSTI_SCAN(16, R); break;                                                                              \
    default: VOSTI_SCAN(32, R); break;                                                                              \
  }
  if (rows == 8) { VOSTI_SCAN_KS(8) } else if (rows == 16) { VOSTI_SCAN_KS(16) } else { VOSTI_SCAN_KS(32) }
#undef VOSTI_SCAN_KS
#undef VOSTI_SCAN
  VOSTI_LAUNCH_CHECK();
}

VOSTI_API int vosti_delta_out(const float* o, const float* gate, const void* w, int w_f32, void* y, int y_f32, int tokens,
                              int heads, int dv, float eps, int w_per_head, cudaStream_t stream) {
  VOSTI_REQUIRE(tokens >= 0 && heads > 0 && dv > 0, "delta_out: bad sizes");
  if (tokens == 0) return VOSTI_OK;
  const int64_t pairs = (int64_t)tokens * heads;
  const unsigned blocks = (unsigned)((pairs + 3) / 4);
  if (y_f32) vosti_launch(delta_out_kernel<float>, dim3(blocks), dim3(128), 0, stream, o, gate, w, w_f32, (float*)y, pairs, dv, eps, heads, w_per_head);
  else vosti_launch(delta_out_kernel<bf16>, dim3(blocks), dim3(128), 0, stream, o, gate, w, w_f32, (bf16*)y, pairs, dv, eps, heads, w_per_head);
  VOSTI_LAUNCH_CHECK();
}

// proj [tokens, stride] (serving type) holds r | k | v | g | a at the given offsets; inner float32
// [tokens, heads * d]; outputs float32 [tokens, heads * d] each.
VOSTI_API int vosti_general_delta_prep(const void* proj, int proj_f32, int stride, int off_r, int off_k, int off_v, int off_g,
                                       int off_a, const float* inner, const void* w0, const void* a_bias, int w_f32,
                                       int heads, int d, int tokens, float* r, float* k, float* v, float* decay, float* unit,
                                       float* removal, float* gate, cudaStream_t stream) {
  VOSTI_REQUIRE(heads > 0 && d > 0 && tokens >= 0, "general_delta_prep: bad sizes");
  if (tokens == 0) return VOSTI_OK;
  GeneralPrepArgs a = {};
  a.proj = proj; a.proj_f32 = proj_f32; a.stride = stride;
  a.off_r = off_r; a.off_k = off_k; a.off_v = off_v; a.off_g = off_g; a.off_a = off_a;
  a.inner = inner; a.w0 = w0; a.a_bias = a_bias; a.w_f32 = w_f32; a.heads = heads; a.d = d;
  a.r = r; a.k = k; a.v = v; a.decay = decay; a.unit = unit; a.removal = removal; a.gate = gate;
  VOSTI_REQUIRE((heads + 3) / 4 <= 65535, "general_delta_prep: too many heads");
  const int size = proj_f32 ? 4 : 2;
  const bool wide = d == 128 && stride % 4 == 0 && (off_r | off_k | off_v | off_g | off_a) % 4 == 0 && reinterpret_cast<uintptr_t>(proj) % (4 * size) == 0 &&
                    ((reinterpret_cast<uintptr_t>(inner) | reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                      reinterpret_cast<uintptr_t>(decay) | reinterpret_cast<uintptr_t>(unit) | reinterpret_cast<uintptr_t>(removal) |
                      reinterpret_cast<uintptr_t>(gate)) & 15) == 0;
  const dim3 grid(tokens, (heads + 3) / 4);
  if (wide && proj_f32) vosti_launch(general_prep_wide_kernel<float>, grid, dim3(128), 0, stream, a);
  else if (wide) vosti_launch(general_prep_wide_kernel<bf16>, grid, dim3(128), 0, stream, a);
  else vosti_launch(general_prep_kernel, grid, dim3(128), 0, stream, a);
  VOSTI_LAUNCH_CHECK();
}

VOSTI_API int vosti_general_delta_scan(const float* r, const float* k, const float* v, const float* decay, const float* unit,
                                       const float* removal, float* out, float* state, int64_t state_stride, const int* cu_q,
                                       const int* state_slots, int num_slots, int requests, int heads, int dk, int dv,
                                       int most, cudaStream_t stream) {
  VOSTI_REQUIRE(heads > 0 && dk > 0 && dv > 0, "general_delta_scan: bad head sizes");
  VOSTI_REQUIRE(dk <= 256, "general_delta_scan: %d key channels (at most 256 are taken)", dk);
  VOSTI_REQUIRE(heads <= 65535, "general_delta_scan: too many heads");
  VOSTI_REQUIRE(state_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0, "general_delta_scan: state slots must be 16-byte aligned");
  if (requests == 0) return VOSTI_OK;
  const int rows = scan_rows(dk), ks = scan_lanes(dk), cols = vosti_delta_scan_columns(requests, heads, dk, dv), threads = cols * ks;
  VOSTI_REQUIRE((dv + cols - 1) / cols <= 65535, "general_delta_scan: too many value channels");
  const dim3 grid(requests, heads, (dv + cols - 1) / cols);
  const size_t smem = 2 * (size_t)(TOKENS * (5 * ks * rows + cols)) * sizeof(float);
#define VOSTI_SCAN(KS, R)                                                                                           \
  do {                                                                                                              \
    static bool configured = false;                                                                                 \
    if (!configured) {                                                                                              \
      cudaFuncSetAttribute(general_scan_kernel<KS, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,                 \
                           (int)(2 * (size_t)(TOKENS * (5 * KS * R + SCAN_THREADS / KS)) * sizeof(float)));          \
      configured = true;                                                                                            \
    }                                                                                                               \
    vosti_launch(general_scan_kernel<KS, R>, grid, dim3(threads), smem, stream, r, k, v, decay, unit, removal, out, \
                 state, state_stride, cu_q, state_slots, num_slots, heads, dk, dv, most);                                 \
  } while (0)
#define VOSTI_SCAN_KS(R)                                                                                            \
  switch (ks) {                                                                                                     \
    case 1: VOSTI_SCAN(1, R); break;                                                                                \
    case 2: VOSTI_SCAN(2, R); break;                                                                                \
    case 4: VOSTI_SCAN(4, R); break;                                                                                \
    case 8: VOSTI_SCAN(8, R); break;                                                                                \
    case 16: VOSTI_SCAN(16, R); break;                                                                              \
    default: VOSTI_SCAN(32, R); break;                                                                              \
  }
  if (rows == 8) { VOSTI_SCAN_KS(8) } else if (rows == 16) { VOSTI_SCAN_KS(16) } else { VOSTI_SCAN_KS(32) }
#undef VOSTI_SCAN_KS
#undef VOSTI_SCAN
  VOSTI_LAUNCH_CHECK();
}

VOSTI_API int vosti_tanh_columns(const void* x, int is_f32, int stride, int offset, int width, void* out, int tokens,
                                 cudaStream_t stream) {
  VOSTI_REQUIRE(tokens >= 0 && width > 0 && offset >= 0 && offset + width <= stride, "tanh_columns: bad sizes");
  if (tokens == 0) return VOSTI_OK;
  const int64_t n = (int64_t)tokens * width;
  const int blocks = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
  if (is_f32) vosti_launch(tanh_columns_kernel<float>, dim3(blocks), dim3(256), 0, stream, (const float*)x, stride, offset, width, (float*)out, (int64_t)tokens);
  else vosti_launch(tanh_columns_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, (const bf16*)x, stride, offset, width, (bf16*)out, (int64_t)tokens);
  VOSTI_LAUNCH_CHECK();
}
