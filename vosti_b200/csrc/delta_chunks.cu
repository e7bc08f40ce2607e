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
//   delta_chunk_run       one block per (request, head, 16 value columns): the chunks one after the other; per
//                         chunk [W; O1] S0 and the state's update, both as 8 x 4 register tiles whose summands
//                         are spread over 8 (4) lanes
//
// The scratch takes 516 floats a token and head (644 in the generalized rule); its caller bounds it and the chunks run in
// rounds. Which steps come here and which go token by token: delta_takes_chunks in ops.py, with both sides' times.
//
// 2,048 tokens of one request, 16 heads of 128: 82 us and 194 us (the token-by-token kernel: 698 us); the
// generalized rule over 1,031 + 700 + 317 tokens: 140 us and 278 us (628 us). The first is bound by shared-memory
// latency at two blocks an SM (issue slots 43 % busy), the second by the shared-memory pipe of the 128 SMs that
// have a block: 16-byte operand reads, the shuffles that deal the sums out, the copies of the next chunks.
//
// The token-by-token kernel waits for a shared-memory read, a chain of multiply-adds and two shuffle reductions
// between any two tokens; here the chain between chunks is two small products over 32 tokens.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int CHUNK = 32, HALF = 16, DK = 128, PITCH = DK + 4, COLS = 16;
constexpr int WO = 2 * CHUNK;                    // W and O1 of a key channel, side by side

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
  float *wo, *ends, *us, *gammas;                // [chunk, head, DK, WO], [.., (2) CHUNK, DK], [.., CHUNK, dv], [.., DK]
};

__device__ __forceinline__ float4 at4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void put4(float* p, float a, float b, float c, float d) { *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d); }
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
    float* const to = a.wo + (place * DK + c) * WO;
    float o4[4], w4[4];
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
      o4[i & 3] = row_sum<i + 1>(MQ + i * CHUNK, w, yg);
      w4[i & 3] = w[i];
      gamma *= g;
      if ((i & 3) == 3) {
        put4(to + i - 3, w4[0], w4[1], w4[2], w4[3]);
        put4(to + CHUNK + i - 3, o4[0], o4[1], o4[2], o4[3]);
      }
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

constexpr int WO_PITCH = WO + 4, S_PITCH = COLS + 4, RUN_THREADS = 256;
template <bool PAIR> constexpr int STAGE_FLOATS = DK * WO_PITCH + (PAIR ? 2 : 1) * CHUNK * (DK + S_PITCH) + DK;
template <bool PAIR> constexpr int RUN_STAGES = PAIR ? 2 : 3;

template <bool PAIR>
__global__ void __launch_bounds__(RUN_THREADS) delta_chunk_run_kernel(ChunkArgs a) {
  extern __shared__ __align__(16) float chunk_shared[];
  constexpr int STAGES = RUN_STAGES<PAIR>, STAGE = STAGE_FLOATS<PAIR>, ROWS = (PAIR ? 2 : 1) * CHUNK;
  float* const S = chunk_shared + STAGES * STAGE;               // [DK][S_PITCH]
  pdl_wait();
  pdl_launch_dependents();
  const int request = a.long_requests[blockIdx.x], h = blockIdx.y, col0 = blockIdx.z * COLS;
  const int slot = a.state_slots[request];
  if (slot < 0 || slot >= a.num_slots) return;
  // the request's chunks in this launch: from chunk `begin` on, or from its first one
  const int chunk0 = a.long_chunk0[blockIdx.x] - a.from, begin = max(0, -chunk0);
  const int start = a.cu_q[request] + begin * CHUNK, n = min(a.cu_q[request + 1] - start, (a.count - chunk0 - begin) * CHUNK);
  if (n <= 0) return;
  const int chunks = (n + CHUNK - 1) / CHUNK;
  const int64_t place0 = (int64_t)chunk0 + begin;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row = (int64_t)a.heads * a.dv;
  float* const state = a.state + (int64_t)slot * a.state_stride + ((int64_t)h * a.dv + col0) * DK;
  for (int i = tid; i < COLS * DK; i += RUN_THREADS) S[(i % DK) * S_PITCH + i / DK] = state[i];

  auto load = [&](int chunk) {
    if (chunk < chunks) {
      float* const wo = chunk_shared + chunk % STAGES * STAGE;
      float* const ends = wo + DK * WO_PITCH;
      float* const uv = ends + ROWS * DK;
      float* const gam = uv + ROWS * S_PITCH;
      const int64_t place = (place0 + chunk) * a.heads + h;
      for (int i = tid; i < DK * (WO / 4); i += RUN_THREADS) {
        const int r = i / (WO / 4), c = (i % (WO / 4)) * 4;
        copy16(wo + r * WO_PITCH + c, a.wo + (place * DK + r) * WO + c);
      }
      for (int i = tid; i < ROWS * (DK / 4); i += RUN_THREADS) copy16(ends + i * 4, a.ends + place * ROWS * DK + i * 4);
      const int r = (tid & 127) / (COLS / 4), c = (tid % (COLS / 4)) * 4;   // 32 rows of 4 words of U, and of v
      if (tid < 128) {
        copy16(uv + r * S_PITCH + c, a.us + (place * CHUNK + r) * a.dv + col0 + c);
      } else if (PAIR) {
        const int t = chunk * CHUNK + r;
        copy16(uv + (CHUNK + r) * S_PITCH + c, a.v + (start + min(t, n - 1)) * row + (int64_t)h * a.dv + col0 + c, t < n);
      }
      if (tid < DK / 4) copy16(gam + tid * 4, a.gammas + place * DK + tid * 4);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) load(i);
  // [W; O1] S: lane = 8 summands' groups x 4 tiles of 8 rows x 4 columns
  const int kg = lane & 7, rt = warp, ct = lane >> 3;
  // the update: lane = 4 groups of tokens x 8 tiles of 8 key channels (4 and 4) x 4 columns
  const int tg = lane >> 3, kt = (warp >> 2) * 8 + (lane & 7), ct2 = warp & 3;
#pragma unroll 1
  for (int chunk = 0; chunk < chunks; ++chunk) {
    load(chunk + STAGES - 1);
    const float* const wo = chunk_shared + chunk % STAGES * STAGE;
    const float* const ends = wo + DK * WO_PITCH;
    float* const uv = const_cast<float*>(ends) + ROWS * DK;
    const float* const gam = uv + ROWS * S_PITCH;
    // this thread's outputs are row rt * 8 + kg: a u (the first 32 rows), or an o, whose first part is out there
    const int i = (rt & 3) * 8 + kg;
    float* const out = a.out + (start + chunk * CHUNK + i) * row + (int64_t)h * a.dv + col0 + ct * 4;
    const bool reads = rt >= 4, writes = reads && chunk * CHUNK + i < n;
    float4 base = make_float4(0.f, 0.f, 0.f, 0.f);
    if (writes) base = at4(out);
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
    __syncthreads();
    float acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
#pragma unroll 2
    for (int s = 0; s < DK / 8; ++s) {
      const int k = s * 8 + kg;
      const float4 a0 = at4(wo + k * WO_PITCH + rt * 8), a1 = at4(wo + k * WO_PITCH + rt * 8 + 4);
      const float4 s0 = at4(S + k * S_PITCH + ct * 4);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, sv[4] = {s0.x, s0.y, s0.z, s0.w};
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r], sv[c], acc[r][c]);
    }
    // the lanes' sums meet while the rows are dealt out: half of what a lane has left goes at every step
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1) {
      const bool upper = kg & half;
#pragma unroll
      for (int r = 0; r < half; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float keep = upper ? acc[r + half][c] : acc[r][c], give = upper ? acc[r][c] : acc[r + half][c];
          acc[r][c] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    if (reads) {
      if (writes) put4(out, base.x + acc[0][0], base.y + acc[0][1], base.z + acc[0][2], base.w + acc[0][3]);
    } else {
      float* const u = uv + i * S_PITCH + ct * 4;
      const float4 u0 = at4(u);
      put4(u, u0.x + acc[0][0], u0.y + acc[0][1], u0.z + acc[0][2], u0.w + acc[0][3]);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
#pragma unroll 2
    for (int s = 0; s < ROWS / 4; ++s) {
      const int j = s * 4 + tg;
      const float4 a0 = at4(ends + j * DK + kt * 4), a1 = at4(ends + j * DK + 64 + kt * 4);
      const float4 s0 = at4(uv + j * S_PITCH + ct2 * 4);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, sv[4] = {s0.x, s0.y, s0.z, s0.w};
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(av[r], sv[c], acc[r][c]);
    }
#pragma unroll
    for (int half = 4; half >= 2; half >>= 1) {
      const bool upper = tg & (half >> 1);
#pragma unroll
      for (int r = 0; r < half; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float keep = upper ? acc[r + half][c] : acc[r][c], give = upper ? acc[r][c] : acc[r + half][c];
          acc[r][c] = keep + __shfl_xor_sync(0xffffffffu, give, half * 4);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int k = (tg >> 1) * 64 + kt * 4 + (tg & 1) * 2 + r;
      const float g = gam[k];
      float* const s = S + k * S_PITCH + ct2 * 4;
      const float4 s0 = at4(s);
      put4(s, fmaf(g, s0.x, acc[r][0]), fmaf(g, s0.y, acc[r][1]), fmaf(g, s0.z, acc[r][2]), fmaf(g, s0.w, acc[r][3]));
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int i = tid; i < COLS * DK; i += RUN_THREADS) state[i] = S[(i % DK) * S_PITCH + i / DK];
}

template <bool PAIR>
int launch_chunks(ChunkArgs a, int chunks, int fit, int longs, cudaStream_t stream) {
  constexpr int prepare_bytes = prepare_floats<PAIR>() * (int)sizeof(float);
  constexpr int run_bytes = (RUN_STAGES<PAIR> * STAGE_FLOATS<PAIR> + DK * S_PITCH) * (int)sizeof(float);
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
    vosti_launch(delta_chunk_run_kernel<PAIR>, dim3(longs, a.heads, a.dv / COLS), dim3(RUN_THREADS), run_bytes, stream, a);
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
