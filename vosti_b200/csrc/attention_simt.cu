// Paged causal attention on the CUDA cores, one warp per (query token, query head), or four rows a warp for portions.
// It serves prompts, portions of prompts and single decoded tokens alike, in float32
// arithmetic for both storage types, and is the float32 path's attention.
//
// What a query sees (kernels/triton_kernels/fattn_paged.py:176-179, 220-221): keys
// 0..position of its own request (with a window w > 0 only keys > position - w); query
// head h reads kv head h * nkv / nq. Scores are scaled by scale * log2(e) and the softmax
// runs online in base 2 over key tiles (:228-246); here a tile is 32 keys aligned to the
// absolute key index, so the order of a row's arithmetic depends on its position only,
// not on how the prompt was cut or what else is in the batch. Unlike the reference's
// kernel the probabilities stay in float32 for P.V.
#include "common.cuh"

namespace {
constexpr int WARPS = 4;
constexpr int MAX_D = 256;
constexpr float LOG2E = 1.4426950408889634f;

template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const T* __restrict__ k, int d);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k, int d) {
  float s = 0.f;
  const float4* k4 = reinterpret_cast<const float4*>(k);
  for (int i = 0; i < d / 4; ++i) {
    const float4 v = k4[i];
    s = fmaf(q[4 * i + 0], v.x, s);
    s = fmaf(q[4 * i + 1], v.y, s);
    s = fmaf(q[4 * i + 2], v.z, s);
    s = fmaf(q[4 * i + 3], v.w, s);
  }
  return s;
}
template <>
__device__ __forceinline__ float dot_row<bf16>(const float* __restrict__ q, const bf16* __restrict__ k, int d) {
  float s = 0.f;
  const uint4* k8 = reinterpret_cast<const uint4*>(k);
  for (int i = 0; i < d / 8; ++i) {
    const uint4 raw = k8[i];
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(p[j]);
      s = fmaf(q[8 * i + 2 * j], f.x, s);
      s = fmaf(q[8 * i + 2 * j + 1], f.y, s);
    }
  }
  return s;
}

// Whether the window of `per` tokens around token t (windows start at multiples of `per`) holds tokens of more than two
// requests; all lanes of a warp ask together (per <= 32).
__device__ __forceinline__ bool crowded(const int* __restrict__ request_of, int t, int per, int tokens) {
  const int lane = threadIdx.x & 31, at = t / per * per + lane;
  const bool starts = lane > 0 && lane < per && at < tokens && request_of[at] != request_of[at - 1];
  return __popc(__ballot_sync(0xffffffffu, starts)) > 1;
}

// `window_tokens` > 0: only the tokens of crowded windows of that many (attention_simt_rows_kernel takes the others)
template <typename T>
__global__ void __launch_bounds__(WARPS * 32)
attention_simt_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                      T* __restrict__ out, const int* __restrict__ positions, const int* __restrict__ request_of,
                      const int* __restrict__ block_table, int max_pages, int page_size, int num_pages,
                      int tokens, int nq, int nkv, int d, float scale_log2, int window, int window_tokens, unsigned* status) {
  extern __shared__ float q_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t wid = (int64_t)blockIdx.x * WARPS + warp;
  if (wid >= (int64_t)tokens * nq) return;
  const int t = (int)(wid / nq), h = (int)(wid % nq);
  if (window_tokens > 0 && !crowded(request_of, t, window_tokens, tokens)) return;
  const int g = h * nkv / nq;
  float* qs = q_smem + warp * d;
  const T* qrow = q + ((int64_t)t * nq + h) * d;
  for (int i = lane; i < d; i += 32) qs[i] = to_f32(qrow[i]);
  __syncwarp();

  const int b = request_of[t];
  const int pos = positions[t];
  const int kstart = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int* table = block_table + (int64_t)b * max_pages;

  float m = -INFINITY, l = 0.f;
  float acc[MAX_D / 32];
#pragma unroll
  for (int i = 0; i < MAX_D / 32; ++i) acc[i] = 0.f;

  for (int j0 = (kstart / 32) * 32; j0 <= pos; j0 += 32) {
    const int j = j0 + lane;
    bool valid = j >= kstart && j <= pos;
    int64_t slot = 0;
    float s = -INFINITY;
    if (valid) {
      const int slot_in_table = j / page_size;
      const int page = slot_in_table < max_pages ? table[slot_in_table] : -1;
      if (page < 0 || page >= num_pages) {
        raise_fault(status, VOSTI_FAULT_PAGE_RANGE);
        valid = false;
      } else {
        slot = ((int64_t)page * nkv + g) * page_size + (j % page_size);   // row of (page, head, offset)
        s = dot_row<T>(qs, k_cache + slot * d, d) * scale_log2;
      }
    }
    const float tile_max = warp_max(s);
    if (tile_max == -INFINITY) continue;  // nothing visible here: state untouched
    const float m_new = fmaxf(m, tile_max);
    const float alpha = exp2f(m - m_new);
    const float p = valid ? exp2f(s - m_new) : 0.f;
    l = l * alpha + warp_sum(p);
#pragma unroll
    for (int i = 0; i < MAX_D / 32; ++i) acc[i] *= alpha;
    const int last = min(31, pos - j0);
    for (int kk = 0; kk <= last; ++kk) {
      const float pk = __shfl_sync(0xffffffffu, p, kk);
      const int64_t sk = __shfl_sync(0xffffffffu, slot, kk);
      if (pk == 0.f) continue;
      const T* vrow = v_cache + sk * d;
#pragma unroll
      for (int i = 0; i < MAX_D / 32; ++i) {
        const int idx = lane + 32 * i;
        if (idx < d) acc[i] = fmaf(pk, to_f32(vrow[idx]), acc[i]);
      }
    }
    m = m_new;
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  T* orow = out + ((int64_t)t * nq + h) * d;
#pragma unroll
  for (int i = 0; i < MAX_D / 32; ++i) {
    const int idx = lane + 32 * i;
    if (idx < d) orow[idx] = from_f32<T>(acc[i] * inv);
  }
}


// The same for portions: a block takes up to ROWS (token, head) rows that read one kv head, TOKENS neighbouring tokens of
// the heads that share it, and stages every tile of 32 keys and values in shared memory once for all of them; a
// warp computes four rows at a time. A row's arithmetic is that of the kernel above, operation by operation: a lane per
// key over the head size in order, the online softmax by tiles of 32 keys, the keys in order. The kernel above read every
// key and value row once per query row, each lane along a row of its own: 384 tokens of 32 heads of 128
// over 8, float32: 500 us, against 146 us here.
// Tokens of several requests in a block are taken request by request, so with `skip_crowded` a block of more than two
// requests leaves its tokens to the kernel above: a request of few tokens costs a block as long as a full one (190 ns a
// key; a warp of the kernel above 380 ns, but side by side). 128 tokens beside 32 single ones at 3,000 keys, 16
// heads of 128, took 21.4 ms served by blocks alone, and 2.3 ms by warps alone.
constexpr int ROWS = 32, ROW_WARPS = 8, PER_WARP = ROWS / ROW_WARPS;

template <typename T, int COLS>                    // COLS: 32-column groups of a head, rounded up
__global__ void __launch_bounds__(ROW_WARPS * 32)
attention_simt_rows_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                           T* __restrict__ out, const int* __restrict__ positions, const int* __restrict__ request_of,
                           const int* __restrict__ block_table, int max_pages, int page_size, int num_pages,
                           int tokens, int nq, int nkv, int d, float scale_log2, int window, int skip_crowded, unsigned* status) {
  extern __shared__ __align__(16) float rows_smem[];
  const int pitch = d + 4;                         // an odd number of 16-byte words (d is a multiple of 16): lanes in different banks
  float* const ks = rows_smem;                     // [32][pitch]
  float* const vs = ks + 32 * pitch;               // [32][d]
  float* const qs = vs + 32 * d;                   // [ROWS][d]
  __shared__ int slots[32];                        // row of (page, head, offset) of the tile's keys, -1: none, -2: a page outside the pool
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = nq / nkv, per_block = ROWS / group;        // tokens of a block
  const int g = blockIdx.y, t_begin = blockIdx.x * per_block, t_end = min(tokens, t_begin + per_block);
  if (skip_crowded && crowded(request_of, t_begin, per_block, tokens)) return;
  for (int i = threadIdx.x; i < (t_end - t_begin) * group * d; i += ROW_WARPS * 32) {
    const int row = i / d, t = t_begin + row / group;
    qs[i] = to_f32(q[((int64_t)t * nq + g * group + row % group) * d + i % d]);
  }
  for (int t0 = t_begin; t0 < t_end;) {
    const int b = request_of[t0];
    int t1 = t0 + 1;                               // tokens t0 .. t1 - 1 are this request's
    while (t1 < t_end && request_of[t1] == b) ++t1;
    const int* const table = block_table + (int64_t)b * max_pages;
    int pos[PER_WARP], kstart[PER_WARP], low = 0x7fffffff, high = -1;
    for (int t = t0; t < t1; ++t) {
      const int p = positions[t];
      low = min(low, window > 0 && p - window + 1 > 0 ? p - window + 1 : 0);
      high = max(high, p);
    }
    float m[PER_WARP], l[PER_WARP], acc[PER_WARP][COLS];
#pragma unroll
    for (int e = 0; e < PER_WARP; ++e) {
      const int t = t_begin + (warp * PER_WARP + e) / group;
      const bool mine = t >= t0 && t < t1;
      pos[e] = mine ? positions[t] : -1;
      kstart[e] = mine && window > 0 && pos[e] - window + 1 > 0 ? pos[e] - window + 1 : 0;
      m[e] = -INFINITY;
      l[e] = 0.f;
#pragma unroll
      for (int i = 0; i < COLS; ++i) acc[e][i] = 0.f;
    }
    for (int j0 = low / 32 * 32; j0 <= high; j0 += 32) {
      __syncthreads();                             // the tile before has been read (and the queries are there)
      if (threadIdx.x < 32) {
        const int j = j0 + threadIdx.x;
        int slot = -1;
        if (j >= low && j <= high) {
          const int index = j / page_size;
          const int page = index < max_pages ? table[index] : -1;
          slot = page < 0 || page >= num_pages ? -2 : (page * nkv + g) * page_size + (j - index * page_size);
        }
        slots[threadIdx.x] = slot;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < 32 * (d / 4); i += ROW_WARPS * 32) {
        const int key = i / (d / 4), c = (i % (d / 4)) * 4;
        const int slot = slots[key];
        float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
        if (slot >= 0) {
          kv = load_four(k_cache + (int64_t)slot * d + c);
          vv = load_four(v_cache + (int64_t)slot * d + c);
        }
        *reinterpret_cast<float4*>(ks + key * pitch + c) = kv;
        *reinterpret_cast<float4*>(vs + key * d + c) = vv;
      }
      __syncthreads();
      const int j = j0 + lane;
      const bool there = slots[lane] >= 0;
      float s[PER_WARP];
#pragma unroll
      for (int e = 0; e < PER_WARP; ++e) s[e] = 0.f;
      const float* const qw = qs + warp * PER_WARP * d;
#pragma unroll 4
      for (int c = 0; c < d; c += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(ks + lane * pitch + c);
#pragma unroll
        for (int e = 0; e < PER_WARP; ++e) {
          const float4 qv = *reinterpret_cast<const float4*>(qw + e * d + c);
          s[e] = fmaf(qv.w, kv.w, fmaf(qv.z, kv.z, fmaf(qv.y, kv.y, fmaf(qv.x, kv.x, s[e]))));
        }
      }
      float p[PER_WARP];
      int last = -1;
#pragma unroll
      for (int e = 0; e < PER_WARP; ++e) {
        const bool visible = j >= kstart[e] && j <= pos[e], valid = visible && there;
        if (visible && !there) raise_fault(status, VOSTI_FAULT_PAGE_RANGE);
        s[e] = valid ? s[e] * scale_log2 : -INFINITY;
        const float tile_max = warp_max(s[e]);
        p[e] = 0.f;
        if (tile_max == -INFINITY) continue;       // nothing visible here: state untouched
        const float m_new = fmaxf(m[e], tile_max);
        const float alpha = exp2f(m[e] - m_new);
        p[e] = valid ? exp2f(s[e] - m_new) : 0.f;
        l[e] = l[e] * alpha + warp_sum(p[e]);
#pragma unroll
        for (int i = 0; i < COLS; ++i) acc[e][i] *= alpha;
        m[e] = m_new;
        last = max(last, min(31, pos[e] - j0));
      }
      for (int kk = 0; kk <= last; ++kk) {
        float v[COLS];
#pragma unroll
        for (int i = 0; i < COLS; ++i) v[i] = lane + 32 * i < d ? vs[kk * d + lane + 32 * i] : 0.f;
#pragma unroll
        for (int e = 0; e < PER_WARP; ++e) {
          const float pk = __shfl_sync(0xffffffffu, p[e], kk);
          if (pk == 0.f) continue;
#pragma unroll
          for (int i = 0; i < COLS; ++i) acc[e][i] = fmaf(pk, v[i], acc[e][i]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < PER_WARP; ++e) {
      if (pos[e] < 0) continue;
      const int row = warp * PER_WARP + e, t = t_begin + row / group;
      const float inv = l[e] > 0.f ? 1.f / l[e] : 0.f;
      T* const orow = out + ((int64_t)t * nq + g * group + row % group) * d;
#pragma unroll
      for (int i = 0; i < COLS; ++i)
        if (lane + 32 * i < d) orow[lane + 32 * i] = from_f32<T>(acc[e][i] * inv);
    }
    t0 = t1;
  }
}
}  // namespace

// q, out: [tokens, nq, d]; caches: [num_pages, nkv, page_size, d];
// block_table: [requests, max_pages]; positions, request_of: int32[tokens]. `way` (the bits are the same): 0 a warp per
// (token, head), 1 blocks of rows that share their keys, 2 blocks where at most two requests meet in one, warps elsewhere.
VOSTI_API int vosti_attention_simt(const void* q, const void* k_cache, const void* v_cache, void* out,
                                   const int* positions, const int* request_of, const int* block_table,
                                   int max_pages, int page_size, int num_pages, int tokens, int way, int nq, int nkv,
                                   int d, float scale, int window, int is_f32, unsigned* status,
                                   cudaStream_t stream) {
  VOSTI_REQUIRE(tokens >= 0 && nq > 0 && nkv > 0 && nq % nkv == 0, "attention: bad head counts nq=%d nkv=%d", nq, nkv);
  VOSTI_REQUIRE(d > 0 && d % 16 == 0 && d <= MAX_D, "attention: head_dim %d must be a multiple of 16 and <= %d", d, MAX_D);
  VOSTI_REQUIRE(page_size > 0 && max_pages > 0 && num_pages > 0, "attention: bad cache geometry");
  VOSTI_REQUIRE(window >= 0, "attention: window must be >= 0 (0 = all keys)");
  if (tokens == 0) return VOSTI_OK;
  // The rows' kernel wants up to 32 heads a kv head and values, too, in whole words.
  VOSTI_REQUIRE(way >= 0 && way <= 2, "attention: unknown way %d", way);
  const int group = nq / nkv;
  int window_tokens = 0;
  if (way > 0 && group <= ROWS && nkv <= 65535 && reinterpret_cast<uintptr_t>(k_cache) % 16 == 0 &&
      reinterpret_cast<uintptr_t>(v_cache) % 16 == 0 && (int64_t)num_pages * nkv * page_size < ((int64_t)1 << 31)) {
    const size_t rows_bytes = ((size_t)32 * (d + 4) + 32 * d + ROWS * d) * sizeof(float);
    constexpr int most = (32 * (MAX_D + 4) + 32 * MAX_D + ROWS * MAX_D) * (int)sizeof(float);
    const dim3 grid((tokens + ROWS / group - 1) / (ROWS / group), nkv);
#define VOSTI_ROWS(T, COLS)                                                                                              \
  do {                                                                                                                   \
    static bool configured = false;                                                                                      \
    if (!configured) {                                                                                                   \
      cudaFuncSetAttribute(attention_simt_rows_kernel<T, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);       \
      configured = true;                                                                                                 \
    }                                                                                                                    \
    attention_simt_rows_kernel<T, COLS><<<grid, ROW_WARPS * 32, rows_bytes, stream>>>((const T*)q, (const T*)k_cache,     \
        (const T*)v_cache, (T*)out, positions, request_of, block_table, max_pages, page_size, num_pages, tokens, nq, nkv, \
        d, scale * LOG2E, window, (int)(way == 2), status);                                                              \
  } while (0)
    if (is_f32) { if (d <= 64) VOSTI_ROWS(float, 2); else if (d <= 128) VOSTI_ROWS(float, 4); else VOSTI_ROWS(float, 8); }
    else { if (d <= 64) VOSTI_ROWS(bf16, 2); else if (d <= 128) VOSTI_ROWS(bf16, 4); else VOSTI_ROWS(bf16, 8); }
#undef VOSTI_ROWS
    if (way == 1) VOSTI_LAUNCH_CHECK();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { vosti_set_error("%s", cudaGetErrorString(e)); return (int)e; }
    window_tokens = ROWS / group;
  }
  const int64_t warps = (int64_t)tokens * nq;
  const int64_t blocks = (warps + WARPS - 1) / WARPS;
  VOSTI_REQUIRE(blocks <= 0x7fffffffLL, "attention: too many (token, head) pairs");
  const size_t smem = (size_t)WARPS * d * sizeof(float);
  if (is_f32)
    attention_simt_kernel<float><<<(unsigned)blocks, WARPS * 32, smem, stream>>>((const float*)q, (const float*)k_cache,
        (const float*)v_cache, (float*)out, positions, request_of, block_table, max_pages, page_size, num_pages,
        tokens, nq, nkv, d, scale * LOG2E, window, window_tokens, status);
  else
    attention_simt_kernel<bf16><<<(unsigned)blocks, WARPS * 32, smem, stream>>>((const bf16*)q, (const bf16*)k_cache,
        (const bf16*)v_cache, (bf16*)out, positions, request_of, block_table, max_pages, page_size, num_pages,
        tokens, nq, nkv, d, scale * LOG2E, window, window_tokens, status);
  VOSTI_LAUNCH_CHECK();
}
