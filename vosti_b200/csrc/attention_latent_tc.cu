// Latent attention of long portions on the 5th-generation tensor cores (tcgen05): a rank of 512, a rotated part of
// 64, pages of a multiple of 16 tokens, bfloat16. Semantics as in attention_latent_mma.cu, which keeps the
// other sizes and the steps whose rows are so few that it cuts the keys into segments.
//
//   grid = (row tiles x 2 column halves, requests), the tiles with most keys first. A CTA takes 128 consecutive
//   (token, head) rows of a request and 256 of the 512 columns of the result: the product of all 512 would fill
//   tensor memory and leave no room for scores, so both halves make the scores (1,152 of the 2,176 multiply-adds issued
//   a key and row; the others are 512 for each of a weight's two terms). Its query rows (144 KB) stay in shared memory, which leaves two stages of 32
//   keys. Roles:
//     * 4 softmax warps, one thread per row: scores from tensor memory, online softmax (base 2, float32, the
//       reference maximum raised lazily), and the weights back to tensor memory as TWO bfloat16 numbers, p = hi + lo,
//       where the second product reads them as its A operand;
//     * 2 loader warps, 16 keys each: nine boxes of 64 elements (eight of the latent, one rotated) straight from the page;
//     * 2 issuing threads: S = Q K^T (M 128, N 32, K 576) and O += P V (M 128, N 256, hi and lo over the same keys; V
//       is the latents' own rows, read MN-major).
//   16 heads over 2,048 tokens: 257 us (73 GFLOP, 146 as issued: 570 TFLOP/s), against 721 us of the mma.sync kernel. What
//   bounds it is the scores' shared-memory traffic: with N = 32 every MMA reads 4 KB of queries for 1 KB of keys.
//   Two score buffers, two weight buffers: the scores of a tile are made while the one before passes the softmax.
//   A key whose latents are not finite reaches the rows of its own 128-row tile that do not see it (a weight of 0 meets it in
//   the product), earlier tokens of its own request, as in the other tensor-core kernels of portions.
#include "common.cuh"
#include "latent.cuh"
#include "mma_util.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace {

constexpr int ROWS = 128, KT = 32, GROUP_KEYS = 16, RANK = 512, ROT = 64, HALF_COLS = RANK / 2;
constexpr int BLOCKS = (RANK + ROT) / 64;               // 64-element blocks of a key
constexpr int STAGES = 2, BLOCK_BYTES = KT * 128, STAGE_BYTES = BLOCKS * BLOCK_BYTES, Q_BYTES = BLOCKS * ROWS * 128;
constexpr int THREADS = 256, LOADER_WARP = 4, MMA_WARP = 6;
constexpr uint32_t TMEM_COLS = 512, S_COL = 0, P_COL = 2 * KT, O_COL = 4 * KT;
constexpr float LOG2E = 1.4426950408889634f;
constexpr size_t SMEM_BYTES = 1024 + Q_BYTES + (size_t)STAGES * STAGE_BYTES;

__global__ void __launch_bounds__(THREADS, 1)
latent_attend_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_c,
                        const __grid_constant__ CUtensorMap map_r, float* __restrict__ out, const int* __restrict__ positions,
                        const int* __restrict__ cu_q, const int* __restrict__ block_table, int max_pages, int page_size,
                        int num_pages, int heads, float scale_log2, int window, const float* __restrict__ sink, unsigned* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* const q_s = smem;                          // [block][128 rows][128 B]
  uint8_t* const k_s = q_s + Q_BYTES;                 // [stage][block][32 keys][128 B]
  __shared__ __align__(8) uint64_t q_full, k_full[STAGES], k_empty[STAGES], edge_bar[KT / GROUP_KEYS];
  __shared__ __align__(8) uint64_t s_full[2], s_empty[2], p_full[2], p_empty[2];
  __shared__ uint32_t tmem_base_holder;
  __shared__ volatile int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  const int b = blockIdx.y, half = blockIdx.x & 1;
  const int q_start = cu_q[b], q_len = cu_q[b + 1] - q_start;
  const int rows_total = q_len * heads;
  const int row0 = ((int)(gridDim.x >> 1) - 1 - (int)(blockIdx.x >> 1)) * ROWS;
  if (row0 >= rows_total) return;
  const int64_t first_row = (int64_t)q_start * heads + row0;
  const int token_lo = row0 / heads, token_hi = min(q_len - 1, (row0 + ROWS - 1) / heads);
  const int first_key = first_visible_key(positions[q_start + token_lo], window), key_end = positions[q_start + token_hi] + 1;
  const int tile_begin = first_key / KT * KT;
  const int tiles = (key_end - tile_begin + KT - 1) / KT;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&q_full), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&k_full[i]), KT / GROUP_KEYS);
      mbar_init(smem_u32(&k_empty[i]), 1);
      mbar_init(smem_u32(&edge_bar[i]), 1);
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&s_empty[i]), 4);
      mbar_init(smem_u32(&p_full[i]), 4);
      mbar_init(smem_u32(&p_empty[i]), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_base_holder), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_holder;
  pdl_launch_dependents();            // after the tensor memory is ours: a dependent must not take it first

  if (warp < LOADER_WARP) {
    // ------------------------------------------------------------ softmax
    const int r = threadIdx.x;                                   // row of the tile and lane of tensor memory
    const bool valid = row0 + r < rows_total;
    const int pos = valid ? positions[q_start + (row0 + r) / heads] : -1;
    const int kstart = valid ? first_visible_key(pos, window) : 0;
    const uint32_t lane_base = tmem_base + ((uint32_t)(warp * 32) << 16);
    const uint32_t o_tmem = lane_base + O_COL;
    // The exponentials are taken against m_run, which follows the true running maximum lazily: only when a tile's
    // maximum exceeds it by more than RESCALE is it raised and the running product scaled down in tensor memory.
    constexpr float RESCALE = 8.f;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int t = 0; t < tiles; ++t) {
      const int key0 = tile_begin + t * KT, buf = t & 1;
      ok = mbar_wait(smem_u32(&s_full[buf]), (t >> 1) & 1, &abort_flag, status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t raw[32];
      tmem_load32(lane_base + S_COL + buf * KT, raw);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_empty[buf]));      // the scores are in registers
      // keys this row does not see
      if (key0 + KT - 1 > pos || key0 < kstart) {
#pragma unroll
        for (int i = 0; i < KT; ++i)
          if (key0 + i > pos || key0 + i < kstart) raw[i] = 0xff800000u;          // -inf
      }
      float part_max[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < KT; ++i) part_max[i & 3] = fmaxf(part_max[i & 3], __uint_as_float(raw[i]));
      const float tile_max = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3])) * scale_log2;
      const bool raise = tile_max > m_run + RESCALE || (m_run == -INFINITY && tile_max > -INFINITY);
      float alpha = 1.f;
      if (raise) {
        alpha = m_run == -INFINITY ? 0.f : fast_exp2(m_run - tile_max);
        m_run = tile_max;
        l_run *= alpha;
      }
      const float safe = m_run == -INFINITY ? 0.f : m_run;
      // this tile's weights may be written once the product of the tile before the last one is complete; rows whose
      // maximum rose also wait for the last product and scale what has run up
      if (t >= 2) ok = mbar_wait(smem_u32(&p_empty[buf]), ((t >> 1) - 1) & 1, &abort_flag, status);
      const bool scales = t >= 1 && __any_sync(0xffffffffu, raise);
      if (scales && ok) ok = mbar_wait(smem_u32(&p_empty[buf ^ 1]), ((t - 1) >> 1) & 1, &abort_flag, status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if (scales) {
#pragma unroll 1
        for (int c0 = 0; c0 < HALF_COLS; c0 += 32) {
          uint32_t v[32];
          tmem_load32(o_tmem + c0, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_store32(o_tmem + c0, v);
        }
      }
      uint32_t p[32];                                            // 16 pairs of hi, then of lo
      float part_sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < KT; i += 2) {
        const float p0 = fast_exp2(fmaf(__uint_as_float(raw[i]), scale_log2, -safe)), p1 = fast_exp2(fmaf(__uint_as_float(raw[i + 1]), scale_log2, -safe));
        part_sum[i & 3] += p0;
        part_sum[(i & 3) + 1] += p1;
        const __nv_bfloat162 hi = __floats2bfloat162_rn(p0, p1);
        const float2 back = __bfloat1622float2(hi);
        p[i >> 1] = *reinterpret_cast<const uint32_t*>(&hi);
        p[16 + (i >> 1)] = pack_bf16(p0 - back.x, p1 - back.y);
      }
      l_run += (part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]);
      tmem_store32(lane_base + P_COL + buf * KT, p);
      tmem_wait_stores();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[buf]));
    }
    // the last product complete means every product is: normalise and store, 32 columns at a time through this
    // warp's part of the query rows' memory, so that the stores are whole rows of 128 bytes
    if (ok) ok = mbar_wait(smem_u32(&p_empty[(tiles - 1) & 1]), ((tiles - 1) >> 1) & 1, &abort_flag, status);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      const float inv = valid ? sink_inverse(m_run, l_run, sink != nullptr ? sink[(row0 + r) % heads] * LOG2E : -INFINITY) : 0.f;
      constexpr int PITCH = 36;
      float* const stage = reinterpret_cast<float*>(q_s) + warp * 32 * PITCH;
      float* const dst = out + (first_row + warp * 32) * RANK + half * HALF_COLS;
      const int rows_here = min(32, rows_total - row0 - warp * 32);
#pragma unroll 1
      for (int c0 = 0; c0 < HALF_COLS; c0 += 32) {
        uint32_t v[32];
        tmem_load32(o_tmem + c0, v);
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<float4*>(stage + lane * PITCH + i) =
              make_float4(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv, __uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int row = i * 4 + (lane >> 3), c = (lane & 7) * 4;
          if (row < rows_here) *reinterpret_cast<float4*>(dst + (int64_t)row * RANK + c0 + c) = *reinterpret_cast<const float4*>(stage + row * PITCH + c);
        }
        __syncwarp();
      }
    }
    tc_fence_before();
  } else if (warp < MMA_WARP) {
    // ------------------------------------------------------------ loaders
    const int w = warp - LOADER_WARP;                    // keys 16 w .. 16 w + 15 of every tile
    if (w == 0 && lane == 0) {
      // (rows past the end of the tensor come as zeros and still count as bytes)
      mbar_expect_tx(smem_u32(&q_full), (uint32_t)Q_BYTES);
      for (int i = 0; i < BLOCKS; ++i) tma_load_2d(smem_u32(q_s + i * (ROWS * 128)), &map_q, i * 64, (int)first_row, smem_u32(&q_full));
    }
    const int* const table = block_table + (int64_t)b * max_pages;
    bool ok = true;
    uint32_t edges = 0;
    for (int t = 0; t < tiles; ++t) {
      const int stage = t & 1;
      if (t >= STAGES) ok = mbar_wait(smem_u32(&k_empty[stage]), ((t >> 1) - 1) & 1, &abort_flag, status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const int lo = tile_begin + t * KT + w * GROUP_KEYS;
      uint8_t* const dst = k_s + stage * STAGE_BYTES + w * GROUP_KEYS * 128;
      int row = -1;
      if (lo + GROUP_KEYS - 1 >= first_key && lo < key_end) {
        const int index = lo / page_size;
        const int page = index < max_pages ? table[index] : -1;
        if (page < 0 || page >= num_pages) raise_fault(status, VOSTI_FAULT_PAGE_RANGE);
        else row = page * page_size + (lo - index * page_size);
      }
      const int keep = row < 0 ? 0 : min(GROUP_KEYS, key_end - lo);     // keys that stay; zeros in the others' place, so
      const bool whole = keep == GROUP_KEYS;                            // that a weight of 0 meets finite values
      const uint32_t bar = whole ? smem_u32(&k_full[stage]) : smem_u32(&edge_bar[w]);
      if (keep > 0) {
        if (lane == 0) mbar_expect_tx(bar, (uint32_t)(BLOCKS * GROUP_KEYS * 128));
        __syncwarp();
        if (lane < BLOCKS)
          tma_load_2d(smem_u32(dst + lane * BLOCK_BYTES), lane < RANK / 64 ? &map_c : &map_r, lane < RANK / 64 ? lane * 64 : 0, row, bar);
      }
      if (!whole) {
        if (keep > 0) {
          ok = mbar_wait(bar, edges & 1, &abort_flag, status);
          ++edges;
        }
        for (int i = lane; i < BLOCKS * GROUP_KEYS * 8; i += 32) {
          const int in_block = i % (GROUP_KEYS * 8);
          if ((in_block >> 3) >= keep)
            *reinterpret_cast<uint4*>(dst + (i / (GROUP_KEYS * 8)) * BLOCK_BYTES + in_block * 16) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&k_full[stage]));
      }
    }
  } else if (lane == 0) {
    // ------------------------------------------------------------ MMA issue: scores, products
    constexpr uint32_t idesc_s = umma_instr_desc(ROWS, KT, false);
    constexpr uint32_t idesc_o = umma_instr_desc(ROWS, HALF_COLS, true);
    bool ok = true;
    if (warp == MMA_WARP) {
      const uint64_t q_desc = smem_desc_sw128(smem_u32(q_s)), k_desc = smem_desc_sw128(smem_u32(k_s));
      ok = mbar_wait(smem_u32(&q_full), 0, &abort_flag, status);
      for (int t = 0; t < tiles && ok; ++t) {
        const int stage = t & 1;
        ok = mbar_wait(smem_u32(&k_full[stage]), (t >> 1) & 1, &abort_flag, status);
        if (ok && t >= 2) ok = mbar_wait(smem_u32(&s_empty[stage]), ((t >> 1) - 1) & 1, &abort_flag, status);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int kb = 0; kb < BLOCKS; ++kb)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16(tmem_base + S_COL + stage * KT, q_desc + (uint64_t)((kb * (ROWS * 128) + ks * 32) >> 4),
                      k_desc + (uint64_t)((stage * STAGE_BYTES + kb * BLOCK_BYTES + ks * 32) >> 4), idesc_s, (kb | ks) ? 1u : 0u);
        umma_commit(smem_u32(&s_full[stage]));
      }
    } else {
      const uint64_t v_desc = smem_desc_sw128_mn(smem_u32(k_s) + half * (HALF_COLS / 64) * BLOCK_BYTES, BLOCK_BYTES);
      for (int t = 0; t < tiles && ok; ++t) {
        const int stage = t & 1;
        ok = mbar_wait(smem_u32(&k_full[stage]), (t >> 1) & 1, &abort_flag, status) &&
             mbar_wait(smem_u32(&p_full[stage]), (t >> 1) & 1, &abort_flag, status);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int part = 0; part < 2; ++part)             // hi, lo
#pragma unroll
          for (int ks = 0; ks < KT / 16; ++ks)
            umma_bf16_ts(tmem_base + O_COL, tmem_base + P_COL + stage * KT + part * (KT / 2) + ks * 8,
                         v_desc + (uint64_t)((stage * STAGE_BYTES + ks * 16 * 128) >> 4), idesc_o, (t | part | ks) ? 1u : 0u);
        umma_commit(smem_u32(&p_empty[stage]));
        umma_commit(smem_u32(&k_empty[stage]));          // (the scores of this stage were complete before its weights came)
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {                                      // what was issued may still be under way
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace

// Whether the tensor-memory kernel takes these sizes.
VOSTI_API int vosti_latent_attend_tc_fits(int rank, int rot, int page_size) {
  return rank == RANK && rot == ROT && page_size > 0 && page_size % GROUP_KEYS == 0;
}

// As vosti_latent_attend_mma without segments; qk holds `tokens` tokens in all.
VOSTI_API int vosti_latent_attend_tc(const void* qk, const void* c_cache, const void* r_cache, float* out, const int* positions,
                                     const int* cu_q, const int* block_table, int max_pages, int page_size, int num_pages,
                                     int requests, int max_q_len, int tokens, int heads, int rank, int rot, float scale, int window,
                                     const float* sink, unsigned* status, cudaStream_t stream) {
  VOSTI_REQUIRE(vosti_latent_attend_tc_fits(rank, rot, page_size), "latent_attend_tc: sizes this kernel does not take");
  VOSTI_REQUIRE(requests >= 0 && requests <= 65535 && heads > 0 && max_pages > 0 && num_pages > 0 && window >= 0, "latent_attend_tc: bad geometry");
  VOSTI_REQUIRE(scale > 0.f, "latent_attend_tc: the score scale must be positive");
  if (requests == 0 || max_q_len <= 0 || tokens == 0) return VOSTI_OK;
  const int64_t rows = (int64_t)tokens * heads, cache_rows = (int64_t)num_pages * page_size;
  VOSTI_REQUIRE(rows < (int64_t)1 << 31 && cache_rows < (int64_t)1 << 31, "latent_attend_tc: too many rows");
  CUtensorMap map_q, map_c, map_r;
  VOSTI_REQUIRE(encode_tensor_map_2d(&map_q, qk, rows, RANK + ROT, ROWS, 64) && cached_tensor_map(c_cache, cache_rows, RANK, GROUP_KEYS, &map_c) &&
                    cached_tensor_map(r_cache, cache_rows, ROT, GROUP_KEYS, &map_r), "latent_attend_tc: cuTensorMapEncodeTiled failed");
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(latent_attend_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    configured = true;
  }
  const int64_t tiles = ((int64_t)max_q_len * heads + ROWS - 1) / ROWS;
  vosti_launch(latent_attend_tc_kernel, dim3((unsigned)(2 * tiles), requests), dim3(THREADS), SMEM_BYTES, stream, map_q, map_c, map_r, out,
               positions, cu_q, block_table, max_pages, page_size, num_pages, heads, scale * LOG2E, window, sink, status);
  VOSTI_LAUNCH_CHECK();
}
