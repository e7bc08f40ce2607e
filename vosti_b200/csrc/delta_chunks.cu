// Long portions of the two delta rules (csrc/delta_rule.cu has the rules and their token-by-token form), in
// chunks of 32 tokens. Everything is float32.
//
// Both rules are, per head, with a decay g_t per key channel,
//     S_t = diag(g_t) S_{t-1} + x_t u_t^T [+ k_t v_t^T],    u_t = init_t - s_t b_t^T S_{t-1},    o_t = S_t^T y_t
//   gated:        x = k, b = g * k, s = beta, init = beta v, y = q       (one update vector)
//   generalized:  x = removal, b = unit key, s = 1, init = 0, y = r, and the term k v^T    (PAIR)
// Inside a chunk u is linear in the chunk's start state S0, u = U + W S0, and so is o = O0 + O1 S0, with W and U
// by forward substitution over the chunk's tokens:
//     W_i = -s_i (b_i G_{i-1}) - sum_{j<i} A_ij W_j            G_i = g_0 * .. * g_i
//     U_i = init_i [- sum_{j<i} B_ij v_j] - sum_{j<i} A_ij U_j
//     O_i = sum_{j<=i} Q_ij (W_j | U_j) + (y_i G_i | [sum_{j<=i} R_ij v_j])
//     A_ij = s_i sum_c b_i x_j P_ij, Q_ij = sum_c y_i g_i x_j P_ij (Q_ii = y_i . x_i), P_ij = g_{j+1} * .. * g_{i-1}
//   (B and R: the same with k in x's place), and S_end = G_31 S0 + sum_j (x_j g_{j+1} .. g_31) u_j^T [+ the same of k, v].
// Every product of decays runs forward between two tokens of the chunk, so nothing is divided and nothing
// overflows, whatever the decays: between tokens of one half of the chunk P is multiplied up pair by pair; between
// the halves it splits at the boundary into two factors of at most 1 each, which makes that block a plain product.
//
// Kernels:
//   delta_chunk_prepare   one block per (chunk, head), all side by side: A, Q (B, R), then one thread per key
//                         channel (W, O1) and per value column (U, O0)
//   delta_chunk_run       one block per (request, head, 16 value columns): the chunks one after the other; per chunk
//                         [W; O1] S0 and the state's update on mma.sync, every operand as three bfloat16 terms
//
// The scratch takes 516 floats a token and head (644 in the generalized rule); its caller bounds it and the chunks run in
// rounds. Which steps come here and which go token by token: delta_takes_chunks in ops.py, with both sides' times.
//
// 2,048 tokens of one request, 16 heads of 128, each launch alone: 79 us and 159 us, 224 for both after one another, whose launches
// overlap (the token-by-token kernel: 695 us); the generalized rule over 1,031 + 700 + 317 tokens: 138 us and 215 us, 330 for
// both (648 us). The first is bound by the shared-memory pipe at two blocks an SM.
// The second was too (8 x 4 tiles of multiply-adds with 16-byte operand reads, shuffles, copies: 194 and 281 us); on the tensor
// cores a chunk takes 2.5 us (generalized 3.4), of which its MMAs are 0.7 and the copies that the blocks' SMs take in
// 0.4, the rest is two barriers and the latency between them: tensor cores 37 % and issue slots 43 % busy, shared memory 43 %. (A copy a row by
// cp.async.bulk instead took 2.7 times as long a chunk; four whole ones from a padded scratch as long as it is.)
// tcgen05 would add a commit and a read of tensor memory to each of the two products of the chain, which are
// 64 x 16 x 128 and 128 x 16 x 32.
//
// The token-by-token kernel waits for a shared-memory read, a chain of multiply-adds and two shuffle reductions
// between any two tokens; here the chain between chunks is two small products over 32 tokens.
#include <type_traits>

#include "common.cuh"
#include "mma_util.cuh"

namespace {

constexpr int CHUNK = 32, HALF = 16, DK = 128, PITCH = DK + 4, COLS = 16;
constexpr int WO = 2 * CHUNK;                    // rows of W and of O1, one below the other

struct ChunkArgs {
  const float *x, *y, *g, *b, *k, *v, *beta;     // b and k: the generalized rule's unit and write keys; beta: the gated rule's
  int x_heads, heads, dv;                        // x and y have x_heads heads (gated: the key heads), the others `heads`
  float* out;
  float* state;
  int64_t state_stride;
  const int *cu_q, *state_slots;
  int num_slots;
  const int *chunk_request, *chunk_first;        // per chunk: its request and its first token in the portion
  const int *long_requests, *long_chunk0;        // per long request: its number and its first chunk
  int from, count;                               // this launch's chunks; the scratch holds them, from 0 on
  float *wo, *ends, *us, *gammas;                // [chunk, head, WO, DK], [.., (2) CHUNK, DK], [.., CHUNK, dv], [.., DK]
};

__device__ __forceinline__ float4 at4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }

template <bool PAIR>
constexpr int prepare_floats() {
  // g, x, y rows (and k, b); the matrices; sums under way; the gated rule's decayed halves; beta
  return (PAIR ? 5 : 3) * CHUNK * PITCH + (PAIR ? 4 : 2) * CHUNK * CHUNK + 2048 + (PAIR ? 0 : 2 * HALF * PITCH) + CHUNK;
}

// sum over j < N of m[j] * r[j], four at a time from a 16-byte aligned row
template <int N>
__device__ __forceinline__ float row_sum(const float* m, const float (&r)[CHUNK], float acc) {
#pragma unroll
  for (int j = 0; j + 4 <= N; j += 4) {
    const float4 a = at4(m + j);
    acc = fmaf(a.x, r[j], acc);
    acc = fmaf(a.y, r[j + 1], acc);
    acc = fmaf(a.z, r[j + 2], acc);
    acc = fmaf(a.w, r[j + 3], acc);
  }
#pragma unroll
  for (int j = N / 4 * 4; j < N; ++j) acc = fmaf(m[j], r[j], acc);
  return acc;
}

template <int I, int N, typename F>
__device__ __forceinline__ void each(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    each<I + 1, N>(f);
  }
}

template <bool PAIR>
__global__ void __launch_bounds__(256, 2) delta_chunk_prepare_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float chunk_shared[];
  constexpr int SOURCES = PAIR ? 2 : 1;
  float* const G = chunk_shared;
  float* const X = G + CHUNK * PITCH;
  float* const Y = X + CHUNK * PITCH;
  float* const K = PAIR ? Y + CHUNK * PITCH : X;
  float* const B = PAIR ? K + CHUNK * PITCH : nullptr;
  float* const mats = Y + (PAIR ? 3 : 1) * CHUNK * PITCH;        // A | Q (of x), B | R (of k)
  float* const sums = mats + SOURCES * 2 * CHUNK * CHUNK;        // [2][half][A, Q][16][16]
  float* const extra = sums + 2048;
  // decayed to the boundary between the halves: x (k) of the first half, b of the second, y g of the second
  float* const XE = PAIR ? X : extra;
  float* const BH = PAIR ? B + HALF * PITCH : extra + HALF * PITCH;
  float* const YH = Y + HALF * PITCH;
  float* const sbeta = extra + (PAIR ? 0 : 2 * HALF * PITCH);
  pdl_wait();
  pdl_launch_dependents();
  const int chunk = a.from + blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int request = a.chunk_request[chunk], first = a.chunk_first[chunk];
  const int64_t t0 = a.cu_q[request] + first;
  const int count = min(CHUNK, a.cu_q[request + 1] - a.cu_q[request] - first);
  const int xh = h / (a.heads / a.x_heads);
  for (int i = tid; i < CHUNK * (DK / 4); i += 256) {
    const int row = i / (DK / 4), c = (i % (DK / 4)) * 4;
    const bool there = row < count;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t at_x = ((t0 + row) * a.x_heads + xh) * DK + c, at_h = ((t0 + row) * a.heads + h) * DK + c;
    *reinterpret_cast<float4*>(G + row * PITCH + c) = there ? at4(a.g + at_h) : make_float4(1.f, 1.f, 1.f, 1.f);
    *reinterpret_cast<float4*>(X + row * PITCH + c) = there ? at4(a.x + at_x) : zero;
    *reinterpret_cast<float4*>(Y + row * PITCH + c) = there ? at4(a.y + at_x) : zero;
    if (PAIR) {
      *reinterpret_cast<float4*>(K + row * PITCH + c) = there ? at4(a.k + at_h) : zero;
      *reinterpret_cast<float4*>(B + row * PITCH + c) = there ? at4(a.b + at_h) : zero;
    }
  }
  if (!PAIR && tid < CHUNK) sbeta[tid] = tid < count ? a.beta[(t0 + tid) * a.heads + h] : 0.f;
  __syncthreads();

  // pairs inside a half: a warp takes a half and 32 channels, a lane row i of the half and 16 of the channels
#pragma unroll 1
  for (int source = 0; source < SOURCES; ++source) {
    const float* const src = source == 0 ? X : K;
    const int half = warp & 1, quarter = warp >> 1, i = lane & 15, row = half * HALF + i;
    float sa[HALF], sq[HALF], diagonal = 0.f;
#pragma unroll
    for (int j = 0; j < HALF; ++j) { sa[j] = 0.f; sq[j] = 0.f; }
#pragma unroll 1
    for (int c4 = 0; c4 < 4; ++c4) {
      const int c = quarter * 32 + (lane >> 4) * 16 + c4 * 4;
      const float4 gi = at4(G + row * PITCH + c), yi = at4(Y + row * PITCH + c);
      const float4 bi = PAIR ? at4(B + row * PITCH + c) : mul4(gi, at4(X + row * PITCH + c));
      const float4 yw = mul4(yi, gi);
      diagonal = dot4(yi, at4(src + row * PITCH + c), diagonal);
      float4 p = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
      for (int j = HALF - 2; j >= 0; --j) {
        const float4 xj = at4(src + (half * HALF + j) * PITCH + c), gn = at4(G + (half * HALF + j + 1) * PITCH + c);
        const float4 next = mul4(p, gn);
        const bool past = j < i - 1;
        p.x = past ? next.x : 1.f;
        p.y = past ? next.y : 1.f;
        p.z = past ? next.z : 1.f;
        p.w = past ? next.w : 1.f;
        const float4 term = mul4(p, xj);
        sa[j] = dot4(bi, term, sa[j]);
        sq[j] = dot4(yw, term, sq[j]);
      }
    }
    diagonal += __shfl_xor_sync(0xffffffffu, diagonal, 16);
#pragma unroll
    for (int j = 0; j < HALF; ++j) {
      sa[j] += __shfl_xor_sync(0xffffffffu, sa[j], 16);
      sq[j] += __shfl_xor_sync(0xffffffffu, sq[j], 16);
      if (j >= i) { sa[j] = 0.f; sq[j] = j == i ? diagonal : 0.f; }
    }
    // lanes of the lower 16 keep A, the others Q; the channels' quarters add up in two rounds
    float* const mine = sums + (((quarter & 1) * 2 + half) * 2 + (lane >> 4)) * HALF * HALF + i * HALF;
#pragma unroll
    for (int round = 1; round >= 0; --round) {
      if (quarter >> 1 == round) {
#pragma unroll
        for (int j = 0; j < HALF; j += 4) {
          float4 v = lane < 16 ? make_float4(sa[j], sa[j + 1], sa[j + 2], sa[j + 3]) : make_float4(sq[j], sq[j + 1], sq[j + 2], sq[j + 3]);
          if (round == 0) {
            const float4 old = at4(mine + j);
            v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
          }
          *reinterpret_cast<float4*>(mine + j) = v;
        }
      }
      __syncthreads();
    }
    for (int e = tid; e < 2 * 2 * HALF * HALF; e += 256) {
      const int hf = e >> 9, mat = (e >> 8) & 1, ii = (e >> 4) & 15, jj = e & 15, r = hf * HALF + ii;
      float v = sums[e] + sums[1024 + e];
      if (!PAIR && mat == 0) v *= sbeta[r];
      mats[((source * 2 + mat) * CHUNK + r) * CHUNK + hf * HALF + jj] = v;
    }
    __syncthreads();
  }

  // decays to the boundary, one channel a thread
  {
    const int c = tid & (DK - 1);
    float p = 1.f;
    if (tid < DK) {
      for (int j = HALF - 1; j >= 0; --j) {
        XE[j * PITCH + c] = X[j * PITCH + c] * p;
        if (PAIR) K[j * PITCH + c] *= p;
        p *= G[j * PITCH + c];
      }
    } else {
      for (int i = 0; i < HALF; ++i) {
        const int row = HALF + i;
        const float g = G[row * PITCH + c];
        BH[i * PITCH + c] = (PAIR ? B[row * PITCH + c] : g * X[row * PITCH + c]) * p;
        YH[i * PITCH + c] = Y[row * PITCH + c] * g * p;
        p *= g;
      }
    }
  }
  __syncthreads();
  // pairs across the halves: 2 x 2 tiles of both matrices a thread, the channels over 4 lanes
#pragma unroll 1
  for (int source = 0; source < SOURCES; ++source) {
    const float* const xe = source == 0 ? XE : K;
    const int part = tid & 3, ti = (tid >> 2) & 7, tj = tid >> 5;
    float m[2][2][2];
#pragma unroll
    for (int e = 0; e < 8; ++e) m[e >> 2][(e >> 1) & 1][e & 1] = 0.f;
#pragma unroll 2
    for (int c = part * 4; c < DK; c += 16) {
      float4 bi[2], yi[2], xj[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        bi[e] = at4(BH + (ti + 8 * e) * PITCH + c);
        yi[e] = at4(YH + (ti + 8 * e) * PITCH + c);
        xj[e] = at4(xe + (tj + 8 * e) * PITCH + c);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          m[0][e][f] = dot4(bi[e], xj[f], m[0][e][f]);
          m[1][e][f] = dot4(yi[e], xj[f], m[1][e][f]);
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float v = m[e >> 2][(e >> 1) & 1][e & 1];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      const int r = HALF + ti + 8 * ((e >> 1) & 1), j = tj + 8 * (e & 1);
      if (!PAIR && e < 4) v *= sbeta[r];
      if ((e & 3) == part) mats[((source * 2 + (e >> 2)) * CHUNK + r) * CHUNK + j] = v;
    }
  }
  __syncthreads();

  const float* const MA = mats;
  const float* const MQ = mats + CHUNK * CHUNK;
  const int64_t place = (int64_t)blockIdx.x * a.heads + h;
  if (tid < DK) {
    const int c = tid;
    float w[CHUNK], gamma = 1.f, first_half = 1.f;
    float* const to = a.wo + place * WO * DK + c;
    each<0, CHUNK>([&](auto index) {
      constexpr int i = decltype(index)::value;
      if (i == HALF) first_half = gamma;
      const float g = G[i * PITCH + c];
      float bg, yg;                                              // b_i G_{i-1}, y_i G_i
      if (i < HALF) {
        bg = (PAIR ? B[i * PITCH + c] : g * X[i * PITCH + c]) * gamma;
        yg = Y[i * PITCH + c] * g * gamma;
      } else {
        bg = BH[(i - HALF) * PITCH + c] * first_half;
        yg = YH[(i - HALF) * PITCH + c] * first_half;
      }
      if (!PAIR) bg *= sbeta[i];
      w[i] = -row_sum<i>(MA + i * CHUNK, w, bg);
      to[i * DK] = w[i];
      to[(CHUNK + i) * DK] = row_sum<i + 1>(MQ + i * CHUNK, w, yg);
      gamma *= g;
    });
    a.gammas[place * DK + c] = gamma;
    // x (and k) decayed to the chunk's end
    float* const end = a.ends + place * SOURCES * CHUNK * DK + c;
    float tail = 1.f;
#pragma unroll 4
    for (int j = CHUNK - 1; j >= 0; --j) {
      end[j * DK] = X[j * PITCH + c] * tail;
      if (PAIR) end[(CHUNK + j) * DK] = K[j * PITCH + c] * tail;
      if (!PAIR || j >= HALF) tail *= G[j * PITCH + c];          // (PAIR: the first half is decayed to the boundary already)
    }
  } else {
    const int64_t row = (int64_t)a.heads * a.dv;
    for (int col = tid - DK; col < a.dv; col += DK) {
      const float* const from = a.v + t0 * row + (int64_t)h * a.dv + col;
      float* const out = a.out + t0 * row + (int64_t)h * a.dv + col;
      float* const us = a.us + place * CHUNK * a.dv + col;
      float u[CHUNK], v[CHUNK];
#pragma unroll
      for (int i = 0; i < CHUNK; ++i) v[i] = i < count ? from[i * row] : 0.f;
      each<0, CHUNK>([&](auto index) {
        constexpr int i = decltype(index)::value;
        if (PAIR) {
          u[i] = -row_sum<i>(MA + i * CHUNK, u, row_sum<i>(mats + 2 * CHUNK * CHUNK + i * CHUNK, v, 0.f));
        } else {
          u[i] = -row_sum<i>(MA + i * CHUNK, u, -sbeta[i] * v[i]);
        }
        float o = row_sum<i + 1>(MQ + i * CHUNK, u, 0.f);
        if (PAIR) o = row_sum<i + 1>(mats + 3 * CHUNK * CHUNK + i * CHUNK, v, o);
        us[(int64_t)i * a.dv] = u[i];
        if (i < count) out[i * row] = o;
      });
    }
  }
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there = true) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// Two neighbouring values as three words of two bfloat16 terms, each the upper half of what the terms before it leave: nothing of a
// float32 is lost (an infinity leaves inf - inf: a state that overflows turns into NaN).
__device__ __forceinline__ void split_two(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  auto upper = [](float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); };
  auto both = [](float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); };
  const float xm = x - upper(x), ym = y - upper(y);
  h = both(x, y);
  m = both(xm, ym);
  l = both(xm - upper(xm), ym - upper(ym));
}
__device__ __forceinline__ void mma_terms(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_eight(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
// sum += A B (16 x 16 times 16 x 8), A and B as three terms: the product of the first terms is added rounded to nearest, those of order
// 2^-8 to 2^-24 gather in `small` (truncated terms lean to one side: without the last two the states were up to twice as far
// from 64 bits as a chain of multiply-adds). HALVES: the first terms in two sums of 8, which the tensor core truncates less.
template <bool HALVES>
__device__ __forceinline__ void mma_split(float (&sum)[4], float (&small)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2]) {
  float first[4] = {0.f, 0.f, 0.f, 0.f};
  if (HALVES) {
    float lower[4] = {0.f, 0.f, 0.f, 0.f};
    mma_eight(lower, a[0][0], a[0][1], b[0][0]);
    mma_eight(first, a[0][2], a[0][3], b[0][1]);
#pragma unroll
    for (int e = 0; e < 4; ++e) first[e] += lower[e];
  } else {
    mma_terms(first, a[0], b[0]);
  }
  mma_terms(small, a[2], b[1]);
  mma_terms(small, a[1], b[2]);
  mma_terms(small, a[2], b[0]);
  mma_terms(small, a[1], b[1]);
  mma_terms(small, a[0], b[2]);
  mma_terms(small, a[1], b[0]);
  mma_terms(small, a[0], b[1]);
#pragma unroll
  for (int e = 0; e < 4; ++e) sum[e] += first[e];
}

constexpr int WO_PITCH = DK + 8, END_PITCH = DK + 4, U_PITCH = COLS + 4, RUN_THREADS = 256;
constexpr int SP_PITCH = DK + 8, UP_PITCH = CHUNK + 8;          // bfloat16 of a value column in the state's and the updates' planes
template <bool PAIR> constexpr int STAGE_FLOATS = WO * WO_PITCH + (PAIR ? 2 : 1) * CHUNK * (END_PITCH + U_PITCH) + DK;
template <bool PAIR> constexpr int RUN_STAGES = PAIR ? 2 : 3;
template <bool PAIR> constexpr int RUN_BYTES = RUN_STAGES<PAIR> * STAGE_FLOATS<PAIR> * 4 + 3 * COLS * (SP_PITCH + (PAIR ? 2 : 1) * UP_PITCH) * 2;

template <bool PAIR>
__global__ void __launch_bounds__(RUN_THREADS) delta_chunk_run_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float chunk_shared[];
  constexpr int STAGES = RUN_STAGES<PAIR>, STAGE = STAGE_FLOATS<PAIR>, ROWS = (PAIR ? 2 : 1) * CHUNK;
  uint16_t* const SP = reinterpret_cast<uint16_t*>(chunk_shared + STAGES * STAGE);   // [term][value column][key channel] of the state
  uint16_t* const UP = SP + 3 * COLS * SP_PITCH;                 // [term][value column][token] of u [and of v]
  uint16_t* const VP = UP + 3 * COLS * UP_PITCH;
  pdl_wait();
  pdl_launch_dependents();
  // the longest request's blocks first (three of 1,031, 700 and 317 tokens: 63 chunk times end to end, 76 if they take turns)
  const int cols = a.dv / COLS, longs = blockIdx.x / (a.heads * cols);
  const int request = a.long_requests[longs], h = blockIdx.x / cols % a.heads, col0 = blockIdx.x % cols * COLS;
  const int slot = a.state_slots[request];
  if (slot < 0 || slot >= a.num_slots) return;
  // the request's chunks in this launch: from chunk `begin` on, or from its first one
  const int chunk0 = a.long_chunk0[longs] - a.from, begin = max(0, -chunk0);
  const int start = a.cu_q[request] + begin * CHUNK, n = min(a.cu_q[request + 1] - start, (a.count - chunk0 - begin) * CHUNK);
  if (n <= 0) return;
  const int chunks = (n + CHUNK - 1) / CHUNK;
  const int64_t place0 = (int64_t)chunk0 + begin;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row = (int64_t)a.heads * a.dv;
  float* const state = a.state + (int64_t)slot * a.state_stride + ((int64_t)h * a.dv + col0) * DK;

  auto load = [&](int chunk) {
    if (chunk < chunks) {
      float* const wo = chunk_shared + chunk % STAGES * STAGE;
      float* const ends = wo + WO * WO_PITCH;
      float* const uv = ends + ROWS * END_PITCH;
      float* const gam = uv + ROWS * U_PITCH;
      const int64_t place = (place0 + chunk) * a.heads + h;
      for (int i = tid; i < WO * (DK / 4); i += RUN_THREADS) {
        const int r = i / (DK / 4), c = (i % (DK / 4)) * 4;
        copy16(wo + r * WO_PITCH + c, a.wo + place * WO * DK + i * 4);
      }
      for (int i = tid; i < ROWS * (DK / 4); i += RUN_THREADS) {
        const int r = i / (DK / 4), c = (i % (DK / 4)) * 4;
        copy16(ends + r * END_PITCH + c, a.ends + place * ROWS * DK + i * 4);
      }
      const int r = (tid & 127) / (COLS / 4), c = (tid % (COLS / 4)) * 4;   // 32 rows of 4 words of U, and of v
      if (tid < 128) {
        copy16(uv + r * U_PITCH + c, a.us + (place * CHUNK + r) * a.dv + col0 + c);
      } else if (PAIR) {
        const int t = chunk * CHUNK + r;
        copy16(uv + (CHUNK + r) * U_PITCH + c, a.v + (start + min(t, n - 1)) * row + (int64_t)h * a.dv + col0 + c, t < n);
      }
      if (tid < DK / 4) copy16(gam + tid * 4, a.gammas + place * DK + tid * 4);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // Products are transposed: value columns on a tile's 16 rows, so that a warp splits only what it alone multiplies. A lane's results
  // are columns g and g + 8 at two neighbouring places (2 t, 2 t + 1) of the other side.
  const int g = lane >> 2, t = lane & 3;
  const int tile_row = lane & 15, tile_k = (lane >> 4) * 8;      // this lane's row of an `ldmatrix` tile
  const int rows0 = warp * 8 + 2 * t;                            // of [W; O1]: a u (the first 32), or an o, whose first part is out there
  auto terms = [&](const uint16_t* planes, int pitch, int k0, uint32_t (&r)[3][4]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) ldmatrix_x4(r[p], smem_addr(planes + (p * COLS + tile_row) * pitch + k0 + tile_k));
  };
  uint32_t wo_terms[DK / 16][3][2];
  auto split_wo = [&](const float* wo, int ks) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 v = *reinterpret_cast<const float2*>(wo + (warp * 8 + g) * WO_PITCH + ks * 16 + e * 8 + 2 * t);
      split_two(v.x, v.y, wo_terms[ks][0][e], wo_terms[ks][1][e], wo_terms[ks][2][e]);
    }
  };
  float S[2][4];                                                 // [8 key channels each]
  auto publish = [&]() {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t term[3];
        split_two(S[nt][2 * e], S[nt][2 * e + 1], term[0], term[1], term[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p)
          *reinterpret_cast<uint32_t*>(SP + (p * COLS + g + 8 * e) * SP_PITCH + warp * 16 + nt * 8 + 2 * t) = term[p];
      }
  };
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 v = *reinterpret_cast<const float2*>(state + (g + 8 * e) * DK + warp * 16 + nt * 8 + 2 * t);
      S[nt][2 * e] = v.x;
      S[nt][2 * e + 1] = v.y;
    }
  publish();
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) load(i);
  const int i0 = rows0 & (CHUNK - 1);
  float base[4] = {0.f, 0.f, 0.f, 0.f};                          // (an o's first part is asked for a chunk ahead)
  auto ask = [&](int chunk) {
    const float* const out = a.out + (start + chunk * CHUNK + i0) * row + (int64_t)h * a.dv + col0 + g;
    const int left = n - chunk * CHUNK - i0;                     // this lane's tokens that there are: left of two
#pragma unroll
    for (int e = 0; e < 4; ++e) base[e] = (e & 1) < left ? out[(e & 1) * row + (e >> 1) * 8] : 0.f;
  };
  if (warp >= 4) ask(0);
  asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
  __syncthreads();
#pragma unroll
  for (int ks = 0; ks < DK / 16; ++ks) split_wo(chunk_shared, ks);
#pragma unroll 1
  for (int chunk = 0; chunk < chunks; ++chunk) {
    load(chunk + STAGES - 1);
    const float* const wo = chunk_shared + chunk % STAGES * STAGE;
    const float* const ends = wo + WO * WO_PITCH;
    const float* const uv = ends + ROWS * END_PITCH;
    const float* const gam = uv + ROWS * U_PITCH;
    if (warp < 4) {
#pragma unroll
      for (int e = 0; e < 4; ++e) base[e] = uv[(i0 + (e & 1)) * U_PITCH + g + (e >> 1) * 8];
    }
    if (PAIR) {
      const int c = tid & (COLS - 1), j = (tid / COLS) * 2;
      uint32_t term[3];
      split_two(uv[(CHUNK + j) * U_PITCH + c], uv[(CHUNK + j + 1) * U_PITCH + c], term[0], term[1], term[2]);
#pragma unroll
      for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(VP + (p * COLS + c) * UP_PITCH + j) = term[p];
    }
    // [W; O1] S
    uint32_t end_terms[2][ROWS / 16][3][2];
    float sum[4] = {0.f, 0.f, 0.f, 0.f}, small[4][4];
#pragma unroll
    for (int e = 0; e < 16; ++e) small[e >> 2][e & 3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t s_terms[3][4];
      terms(SP, SP_PITCH, ks * 16, s_terms);
      mma_split<false>(sum, small[ks & 3], s_terms, wo_terms[ks]);
      // beside it: the update's weights, and (where three stages fit) the next chunk's [W; O1]
#pragma unroll
      for (int piece = ks * (ROWS / 32); piece < (ks + 1) * (ROWS / 32); ++piece) {
        const int nt = piece & 1, e = (piece >> 1) & 1, ke = piece >> 2;
        const float* const from = ends + (ke * 16 + e * 8 + 2 * t) * END_PITCH + warp * 16 + nt * 8 + g;
        split_two(from[0], from[END_PITCH], end_terms[nt][ke][0][e], end_terms[nt][ke][1][e], end_terms[nt][ke][2][e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[e] = base[e] + (sum[e] + ((small[0][e] + small[1][e]) + (small[2][e] + small[3][e])));
    if (warp < 4) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t term[3];
        split_two(sum[2 * e], sum[2 * e + 1], term[0], term[1], term[2]);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(UP + (p * COLS + g + 8 * e) * UP_PITCH + i0) = term[p];
      }
    } else {
      float* const out = a.out + (start + chunk * CHUNK + i0) * row + (int64_t)h * a.dv + col0 + g;
      const int left = n - chunk * CHUNK - i0;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if ((e & 1) < left) out[(e & 1) * row + (e >> 1) * 8] = sum[e];
      ask(chunk + 1);
    }
    if (STAGES > 2) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");    // (the next chunk is here)
    __syncthreads();
    // the state's decay and update
    float add[2][4], low[2][2][4];
#pragma unroll
    for (int e = 0; e < 8; ++e) add[e >> 2][e & 3] = low[0][e >> 2][e & 3] = low[1][e >> 2][e & 3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < ROWS / 16; ++ks) {
      uint32_t u_terms[3][4];
      terms(ks < 2 ? UP : VP, UP_PITCH, (ks & 1) * 16, u_terms);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        mma_split<true>(add[nt], low[nt][ks & 1], u_terms, end_terms[nt][ks]);
        if (STAGES > 2) {
          split_wo(chunk_shared + (chunk + 1) % STAGES * STAGE, ks * 4 + nt * 2);
          split_wo(chunk_shared + (chunk + 1) % STAGES * STAGE, ks * 4 + nt * 2 + 1);
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // what is lost in g S and in its sum with the first terms joins the small ones: one rounding of the state a chunk
        const float decay = gam[warp * 16 + nt * 8 + 2 * t + (e & 1)], kept = decay * S[nt][e], lost = fmaf(decay, S[nt][e], -kept);
        const float whole = kept + add[nt][e], part = whole - kept;
        S[nt][e] = whole + (((kept - (whole - part)) + (add[nt][e] - part)) + (lost + (low[nt][0][e] + low[nt][1][e])));
      }
    publish();
    if (STAGES == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (STAGES == 2) {
#pragma unroll
      for (int ks = 0; ks < DK / 16; ++ks) split_wo(chunk_shared + (chunk + 1) % STAGES * STAGE, ks);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e)
      *reinterpret_cast<float2*>(state + (g + 8 * e) * DK + warp * 16 + nt * 8 + 2 * t) = make_float2(S[nt][2 * e], S[nt][2 * e + 1]);
}

template <bool PAIR>
int launch_chunks(ChunkArgs a, int chunks, int fit, int longs, cudaStream_t stream) {
  constexpr int prepare_bytes = prepare_floats<PAIR>() * (int)sizeof(float);
  constexpr int run_bytes = RUN_BYTES<PAIR>;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(delta_chunk_prepare_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, prepare_bytes);
    cudaFuncSetAttribute(delta_chunk_run_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, run_bytes);
    configured = true;
  }
  for (a.from = 0; a.from < chunks; a.from += fit) {            // (a request's state waits in its slot between two rounds)
    a.count = chunks - a.from < fit ? chunks - a.from : fit;
    vosti_launch(delta_chunk_prepare_kernel<PAIR>, dim3(a.count, a.heads), dim3(256), prepare_bytes, stream, a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { vosti_set_error("%s", cudaGetErrorString(e)); return (int)e; }
    vosti_launch(delta_chunk_run_kernel<PAIR>, dim3((unsigned)((int64_t)longs * a.heads * (a.dv / COLS))), dim3(RUN_THREADS), run_bytes, stream, a);
    e = cudaGetLastError();
    if (e != cudaSuccess) { vosti_set_error("%s", cudaGetErrorString(e)); return (int)e; }
  }
  return VOSTI_OK;
}

}  // namespace

// Whether the chunked kernels take these head sizes, and the floats of scratch a chunk needs.
VOSTI_API int vosti_delta_chunk_fits(int heads, int dk, int dv) {
  return dk == DK && dv > 0 && dv % COLS == 0 && dv / COLS <= 65535 && heads <= 65535;
}
VOSTI_API int64_t vosti_delta_chunk_floats(int heads, int dv, int pair) {
  return (int64_t)heads * (DK * WO + (pair ? 2 : 1) * CHUNK * DK + CHUNK * dv + DK);
}

// The recurrence over the requests `long_requests`. Gated rule: x = k and y = q [tokens, x_heads, 128], beta
// [tokens, heads], b and k null. Generalized rule: x = removal, b = unit, k, y = r (x_heads = heads), beta null.
// `scratch` has room for `fit` chunks: with fewer than there are, they run in rounds of so many (two launches each).
VOSTI_API int vosti_delta_chunks(const float* x, const float* y, const float* decay, const float* b, const float* k, const float* v,
                                 const float* beta, int x_heads, int heads, int dk, int dv, float* out, float* state,
                                 int64_t state_stride, const int* cu_q, const int* state_slots, int num_slots,
                                 const int* chunk_request, const int* chunk_first, int chunks, const int* long_requests,
                                 const int* long_chunk0, int longs, float* scratch, int fit, cudaStream_t stream) {
  VOSTI_REQUIRE(vosti_delta_chunk_fits(heads, dk, dv) && x_heads > 0 && heads % x_heads == 0, "delta_chunks: head sizes it does not take");
  VOSTI_REQUIRE((b == nullptr) == (k == nullptr) && (b == nullptr) == (beta != nullptr), "delta_chunks: one rule or the other");
  VOSTI_REQUIRE(state_stride % 4 == 0 && ((reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) |
                reinterpret_cast<uintptr_t>(decay) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(scratch)) & 15) == 0, "delta_chunks: operands start on 16-byte boundaries");
  if (chunks == 0 || longs == 0) return VOSTI_OK;
  VOSTI_REQUIRE(scratch != nullptr && fit > 0, "delta_chunks: no scratch");
  VOSTI_REQUIRE((int64_t)longs * heads * (dv / COLS) <= 0x7fffffff, "delta_chunks: too many blocks");
  if (fit > chunks) fit = chunks;
  ChunkArgs a = {};
  a.x = x; a.y = y; a.g = decay; a.b = b; a.k = k; a.v = v; a.beta = beta;
  a.x_heads = x_heads; a.heads = heads; a.dv = dv;
  a.out = out; a.state = state; a.state_stride = state_stride;
  a.cu_q = cu_q; a.state_slots = state_slots; a.num_slots = num_slots;
  a.chunk_request = chunk_request; a.chunk_first = chunk_first; a.long_requests = long_requests; a.long_chunk0 = long_chunk0;
  const int64_t places = (int64_t)fit * heads;
  a.wo = scratch;
  a.ends = a.wo + places * DK * WO;
  a.us = a.ends + places * (b != nullptr ? 2 : 1) * CHUNK * DK;
  a.gammas = a.us + places * CHUNK * dv;
  return b != nullptr ? launch_chunks<true>(a, chunks, fit, longs, stream) : launch_chunks<false>(a, chunks, fit, longs, stream);
}
