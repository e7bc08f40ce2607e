// Latent attention of portions with keys and values of every head formed for the step (bfloat16; heads of 128 + 64, values of
// 128). In the latent space (attention_latent_tc.cu) a key costs a head 1,088 multiply-adds a row, here 192 for the
// score and 128 for the sum; forming a key and a value costs 2 x 128 x rank once a key and head, which some tens of
// rows of a request earn back (`ops.latent_forms_heads` has the measured line).
//
//   latent_gather   the latents and rotated key parts of all requests from their pages into dense rows, every request's
//                   rounded up to 128 with zeros, so that a tile of keys never meets another request's.
//   (a product)     k, v = W_uk c, W_uv c of all rows (vosti_gemm_tc_two_terms): k rounded to bfloat16, as the query's latent
//                   form is in the other kernels, v as TWO bfloat16 numbers, v = hi + lo, because the weighted latent they
//                   replace was float32 (and went into its product as two terms).
//   latent_heads    flash attention, roles as in attention_prefill_tc.cu: two row tiles of 128 tokens of one head, a softmax
//                   warpgroup each; one thread loads whole tiles of 64 keys (7 boxes); four threads issue MMAs. The weights
//                   go back to tensor memory as p = hi + lo, the second product's A operand: p_hi v_hi + p_lo v_hi + p_hi v_lo.
//
// A CTA's two row tiles are the request's i-th and i-th last, so that all CTAs walk the same number of keys, or it has one
// where that still leaves no more CTAs than SMs. A tile of 64 keys costs the tensor core 1,152 cycles a row tile (384
// scores, 768 sums) and its softmax thread some 1,000; the keys' 56 KB a tile are what two row tiles share. 2,048 tokens of 16 heads: 64 us
// (in the latent space 265 and two projections), tensor cores 43 % and issue slots 29 % busy on the 128 SMs that have a block.
// (The softmax's 200 registers are moved to it at run time; 8 bytes of the 128 that the launch starts with lie in local memory.)
#include "common.cuh"
#include "latent.cuh"
#include "mma_util.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace {

constexpr int D = 128, ROT = 64, ROWS = 128, ROW_TILES = 2, KT = 64, STAGES = 2, PAD = 128;
constexpr int Q_BLOCKS = (D + ROT) / 64;
constexpr int Q_BYTES = Q_BLOCKS * ROWS * 128;                    // one row tile of queries
constexpr int BLOCK_BYTES = KT * 128;                             // 64 keys x 64 elements
constexpr int V_AT = Q_BLOCKS * BLOCK_BYTES, LO_AT = V_AT + 2 * BLOCK_BYTES, STAGE_BYTES = LO_AT + 2 * BLOCK_BYTES;
constexpr int THREADS = 512, LOADER_WARP = 8, MMA_WARP = 12;
constexpr uint32_t S_COL = 0, P_COL = 2 * KT, O_COL = 4 * KT, TMEM_COLS = 512;
constexpr float LOG2E = 1.4426950408889634f;
constexpr size_t SMEM_BYTES = 1024 + (size_t)ROW_TILES * Q_BYTES + (size_t)STAGES * STAGE_BYTES;

// First dense row of request b: the lengths before it, each rounded up to PAD. All lanes of a warp call.
__device__ __forceinline__ int dense_start(const int* kv_len, int b) {
  int sum = 0;
  for (int i = threadIdx.x & 31; i < b; i += 32) sum += (kv_len[i] + PAD - 1) / PAD * PAD;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

// 16 dense rows a block: grid (rows / 16 of the longest request, requests).
__global__ void __launch_bounds__(128)
latent_gather_kernel(const bf16* __restrict__ c_cache, const bf16* __restrict__ r_cache, const int* __restrict__ kv_len,
                     const int* __restrict__ block_table, int max_pages, int page_size, int num_pages, int rank,
                     bf16* __restrict__ c_out, bf16* __restrict__ r_out, int rows_out, unsigned* status) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.y, key0 = blockIdx.x * 16, keys = kv_len[b];
  if (key0 >= (keys + PAD - 1) / PAD * PAD) return;
  const int row0 = dense_start(kv_len, b) + key0;
  if (row0 + 16 > rows_out) return;                               // (lengths that are not the host's)
  int64_t from = -1;
  if (key0 < keys) {
    const int index = key0 / page_size, page = index < max_pages ? block_table[(int64_t)b * max_pages + index] : -1;
    if (page < 0 || page >= num_pages) {
      if (threadIdx.x == 0) raise_fault(status, VOSTI_FAULT_PAGE_RANGE);
    } else {
      from = (int64_t)page * page_size + (key0 - index * page_size);
    }
  }
  const int words = rank / 8, each = words + ROT / 8;             // 16-byte words of a row
  for (int i = threadIdx.x; i < 16 * each; i += 128) {
    const int r = i / each, w = i % each;
    const bool there = from >= 0 && key0 + r < keys;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (w < words) {
      if (there) v = *(reinterpret_cast<const uint4*>(c_cache + (from + r) * rank) + w);
      *(reinterpret_cast<uint4*>(c_out + (int64_t)(row0 + r) * rank) + w) = v;
    } else {
      if (there) v = *(reinterpret_cast<const uint4*>(r_cache + (from + r) * ROT) + (w - words));
      *(reinterpret_cast<uint4*>(r_out + (int64_t)(row0 + r) * ROT) + (w - words)) = v;
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1)
latent_heads_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                    const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_lo,
                    const __grid_constant__ CUtensorMap map_r, bf16* __restrict__ out, const int* __restrict__ cu_q,
                    const int* __restrict__ kv_len, int heads, int paired, float scale_log2, const float* __restrict__ sink,
                    const HeadGate gate, unsigned* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* const q_s = smem;                          // [row tile][block][128 rows][128 B]
  uint8_t* const kv_s = q_s + ROW_TILES * Q_BYTES;    // [stage]: k 2 blocks, r, v hi 2, v lo 2, each [64 keys][128 B]
  __shared__ __align__(8) uint64_t q_full, kv_full[STAGES], kv_empty[STAGES];
  __shared__ __align__(8) uint64_t s_full[ROW_TILES], s_empty[ROW_TILES], p_full[ROW_TILES], p_empty[ROW_TILES];
  __shared__ uint32_t tmem_base_holder;
  __shared__ volatile int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y, h = blockIdx.x % heads, at = blockIdx.x / heads;
  pdl_wait();
  const int q_start = cu_q[b], q_len = cu_q[b + 1] - q_start, k_len = kv_len[b], shift = k_len - q_len;
  const int row_tiles = (q_len + ROWS - 1) / ROWS;
  const int last = row_tiles - 1 - at;                            // this CTA's row tiles: the at-th last, and the at-th
  if (last < 0 || (paired && last < at)) return;
  const int tile_of[ROW_TILES] = {last, paired && last > at ? at : -1};
  int tiles_of[ROW_TILES];
#pragma unroll
  for (int w = 0; w < ROW_TILES; ++w)
    tiles_of[w] = tile_of[w] < 0 ? 0 : (shift + min(q_len, (tile_of[w] + 1) * ROWS) + KT - 1) / KT;
  const int tiles = tiles_of[0];                                  // (never fewer than the other's)

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&q_full), 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&kv_full[s]), 1);
      mbar_init(smem_u32(&kv_empty[s]), ROW_TILES);
    }
    for (int i = 0; i < ROW_TILES; ++i) {
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
    // ------------------------------------------------------------ softmax and accumulation
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    const int wg = warp >> 2, r = threadIdx.x & 127;             // its row tile; row of the tile and lane of tensor memory
    const int my_tiles = wg ? tiles_of[1] : tiles_of[0];
    const int token = (wg ? tile_of[1] : tile_of[0]) * ROWS + r;
    const bool valid = my_tiles > 0 && token < q_len;
    const int pos = valid ? shift + token : -1;                  // -1: no key is visible, nothing is written
    const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s_tmem = lane_base + S_COL + wg * KT, p_tmem = lane_base + P_COL + wg * KT, o_tmem = lane_base + O_COL + wg * D;
    // The exponentials are taken against m_run, which follows the true running maximum lazily: only when a tile's
    // maximum exceeds it by more than RESCALE is it raised and the running product scaled down in tensor memory.
    constexpr float RESCALE = 8.f;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int t = 0; t < my_tiles; ++t) {
      const int key0 = t * KT;
      ok = mbar_wait(smem_u32(&s_full[wg]), t & 1, &abort_flag, status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t raw[2][32];
      tmem_load32_async(s_tmem, raw[0]);
      tmem_load32_async(s_tmem + 32, raw[1]);
      tmem_wait_loads();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_empty[wg]));       // the scores are in registers
      if (key0 + KT - 1 > pos) {
#pragma unroll
        for (int i = 0; i < KT; ++i)
          if (key0 + i > pos) raw[i >> 5][i & 31] = 0xff800000u;                  // -inf
      }
      float part_max[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < KT; ++i) part_max[i & 3] = fmaxf(part_max[i & 3], __uint_as_float(raw[i >> 5][i & 31]));
      const float tile_max = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3])) * scale_log2;
      const bool raise = tile_max > m_run + RESCALE || (m_run == -INFINITY && tile_max > -INFINITY);
      float alpha = 1.f;
      if (raise) {
        alpha = m_run == -INFINITY ? 0.f : fast_exp2(m_run - tile_max);
        m_run = tile_max;
        l_run *= alpha;
      }
      const float safe = m_run == -INFINITY ? 0.f : m_run;
      float part_sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int half = 0; half < 2; ++half) {                     // 32 scores become 16 pairs of hi and 16 of lo in place
        uint32_t lo[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(raw[half][i]), scale_log2, -safe));
          const float p1 = fast_exp2(fmaf(__uint_as_float(raw[half][i + 1]), scale_log2, -safe));
          part_sum[i & 3] += p0;
          part_sum[(i & 3) + 1] += p1;
          const __nv_bfloat162 hi = __floats2bfloat162_rn(p0, p1);
          const float2 back = __bfloat1622float2(hi);
          raw[half][i >> 1] = *reinterpret_cast<const uint32_t*>(&hi);
          lo[i >> 1] = pack_bf16(p0 - back.x, p1 - back.y);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) raw[half][16 + i] = lo[i];
      }
      l_run += (part_sum[0] + part_sum[1]) + (part_sum[2] + part_sum[3]);
      // the weights' place is free, and the running product complete, once the product of the tile before is
      if (t >= 1) ok = mbar_wait(smem_u32(&p_empty[wg]), (t - 1) & 1, &abort_flag, status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      if (t >= 1 && __any_sync(0xffffffffu, raise)) {
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t v[32];
          tmem_load32(o_tmem + c0, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_store32(o_tmem + c0, v);
        }
      }
      tmem_store32(p_tmem, raw[0]);                              // keys 0..31: hi, lo; keys 32..63: hi, lo
      tmem_store32(p_tmem + 32, raw[1]);
      tmem_wait_stores();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[wg]));
    }
    if (my_tiles > 0) {
      if (ok) ok = mbar_wait(smem_u32(&p_empty[wg]), (my_tiles - 1) & 1, &abort_flag, status);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
        float inv = valid ? sink_inverse(m_run, l_run, sink != nullptr ? sink[h] * LOG2E : -INFINITY) : 0.f;
        const int t_out = q_start + token;
        if (valid && gate.per_element == nullptr) inv *= gate.at(t_out, h, 0, heads, D);
        bf16* const dst = out + ((int64_t)t_out * heads + h) * D;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t v[32];
          tmem_load32(o_tmem + c0, v);                           // (all lanes of the warp take part)
          if (!valid) continue;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) y[e] = __uint_as_float(v[8 * c + e]) * inv;
            if (gate.per_element != nullptr) {
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                const float2 g = gate.at_pair(t_out, h, c0 + 8 * c + e, heads, D);
                y[e] *= g.x;
                y[e + 1] *= g.y;
              }
            }
            *reinterpret_cast<uint4*>(dst + c0 + 8 * c) =
                make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
          }
        }
      }
    }
    tc_fence_before();
  } else if (warp < MMA_WARP) {
    // ------------------------------------------------------------ loader
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == LOADER_WARP) {
      const int start = dense_start(kv_len, b);
      if (lane == 0) {
        // (rows past the end of the step come as zeros and still count as bytes, another request's are never used)
        mbar_expect_tx(smem_u32(&q_full), (uint32_t)((tiles_of[1] > 0 ? 2 : 1) * Q_BYTES));
        for (int w = 0; w < ROW_TILES; ++w) {
          if (tiles_of[w] == 0) continue;
          const int row = q_start + tile_of[w] * ROWS;
          for (int i = 0; i < D / 64; ++i)
            tma_load_2d(smem_u32(q_s + w * Q_BYTES + i * (ROWS * 128)), &map_q, h * (D + ROT) + i * 64, row, smem_u32(&q_full));
          tma_load_2d(smem_u32(q_s + w * Q_BYTES + (D / 64) * (ROWS * 128)), &map_qr, h * ROT, row, smem_u32(&q_full));
        }
        bool ok = true;
        for (int t = 0; t < tiles && ok; ++t) {
          const int stage = t % STAGES;
          if (t >= STAGES) ok = mbar_wait(smem_u32(&kv_empty[stage]), ((t / STAGES) - 1) & 1, &abort_flag, status);
          if (!ok) break;
          const uint32_t bar = smem_u32(&kv_full[stage]), dst = smem_u32(kv_s + stage * STAGE_BYTES);
          const int row = start + t * KT;
          mbar_expect_tx(bar, (uint32_t)STAGE_BYTES);
          for (int i = 0; i < 2; ++i) {
            tma_load_2d(dst + i * BLOCK_BYTES, &map_kv, h * D + i * 64, row, bar);
            tma_load_2d(dst + V_AT + i * BLOCK_BYTES, &map_kv, (heads + h) * D + i * 64, row, bar);
            tma_load_2d(dst + LO_AT + i * BLOCK_BYTES, &map_lo, h * D + i * 64, row, bar);
          }
          tma_load_2d(dst + 2 * BLOCK_BYTES, &map_r, 0, row, bar);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ MMA issue
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    // four issuing threads, one per warp: scores of row tile 0, of row tile 1, products of row tile 0, of row tile 1
    const int role = warp - MMA_WARP, wg = role & 1;
    const int my_tiles = wg ? tiles_of[1] : tiles_of[0];
    constexpr uint32_t idesc_s = umma_instr_desc(ROWS, KT, false);
    constexpr uint32_t idesc_o = umma_instr_desc(ROWS, D, true);
    bool ok = true;
    auto arrived = [&](uint64_t* bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, &abort_flag, status)) != 0;
    };
    if (role < 2) {
      const uint64_t q_desc = smem_desc_sw128(smem_u32(q_s) + wg * Q_BYTES), k_desc = smem_desc_sw128(smem_u32(kv_s));
      if (my_tiles > 0) ok = arrived(&q_full, 0);
      for (int t = 0; t < my_tiles && ok; ++t) {
        const int stage = t % STAGES;
        ok = arrived(&kv_full[stage], (t / STAGES) & 1);
        if (ok && t >= 1) ok = arrived(&s_empty[wg], (t - 1) & 1);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kb = 0; kb < Q_BLOCKS; ++kb)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_bf16(tmem_base + S_COL + wg * KT, q_desc + (uint64_t)((kb * (ROWS * 128) + ks * 32) >> 4),
                        k_desc + (uint64_t)((stage * STAGE_BYTES + kb * BLOCK_BYTES + ks * 32) >> 4), idesc_s, (kb | ks) ? 1u : 0u);
          umma_commit(smem_u32(&s_full[wg]));
        }
        __syncwarp();
      }
    } else {
      const uint64_t v_desc = smem_desc_sw128_mn(smem_u32(kv_s) + V_AT, BLOCK_BYTES);
      for (int t = 0; t < tiles && ok; ++t) {
        const int stage = t % STAGES;
        ok = arrived(&kv_full[stage], (t / STAGES) & 1);
        if (!ok) break;
        if (t >= my_tiles) {                            // the other row tile's alone: given back as soon as it is here
          if (lane == 0) mbar_arrive(smem_u32(&kv_empty[stage]));
          continue;
        }
        ok = arrived(&p_full[wg], t & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t o = tmem_base + O_COL + wg * D, p = tmem_base + P_COL + wg * KT;
        const uint64_t hi = v_desc + (uint64_t)((stage * STAGE_BYTES) >> 4), lo = hi + (uint64_t)((LO_AT - V_AT) >> 4);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < KT / 16; ++ks) {
            const uint32_t p_hi = p + (ks >> 1) * 32 + (ks & 1) * 8, p_lo = p_hi + 16;
            const uint64_t step = (uint64_t)((ks * 16 * 128) >> 4);
            umma_bf16_ts(o, p_lo, hi + step, idesc_o, (t | ks) ? 1u : 0u);
            umma_bf16_ts(o, p_hi, lo + step, idesc_o, 1u);
            umma_bf16_ts(o, p_hi, hi + step, idesc_o, 1u);
          }
          umma_commit(smem_u32(&p_empty[wg]));
          umma_commit(smem_u32(&kv_empty[stage]));        // (the scores of this stage were complete before its weights came)
        }
        __syncwarp();
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

// Whether the kernels take these sizes (`q_width`: elements of a row of the projection that holds the queries first).
VOSTI_API int vosti_latent_heads_fits(int dim, int rot, int dv, int rank, int page_size, int q_width) {
  return dim == D && dv == D && rot == ROT && rank >= 64 && rank % 8 == 0 && page_size > 0 && page_size % 16 == 0 && q_width % 8 == 0;
}

// Dense latents [rows, rank] and rotated parts [rows, 64] of all requests, kv_len[b] keys each rounded up to 128 rows (zeros);
// `rows` is their sum, max_kv_len the longest.
VOSTI_API int vosti_latent_gather(const void* c_cache, const void* r_cache, const int* kv_len, const int* block_table, int max_pages,
                                  int page_size, int num_pages, int requests, int max_kv_len, int rank, int rot, void* c_out,
                                  void* r_out, int rows, unsigned* status, cudaStream_t stream) {
  VOSTI_REQUIRE(rot == ROT && rank % 8 == 0 && page_size > 0 && page_size % 16 == 0 && max_pages > 0 && num_pages > 0, "latent_gather: bad geometry");
  VOSTI_REQUIRE(requests >= 0 && requests <= 65535, "latent_gather: too many requests for one launch");
  VOSTI_REQUIRE((reinterpret_cast<uintptr_t>(c_cache) | reinterpret_cast<uintptr_t>(r_cache)) % 16 == 0, "latent_gather: caches must be 16-byte aligned");
  if (requests == 0 || max_kv_len <= 0) return VOSTI_OK;
  vosti_launch(latent_gather_kernel, dim3((max_kv_len + PAD - 1) / PAD * (PAD / 16), requests), dim3(128), 0, stream, (const bf16*)c_cache,
               (const bf16*)r_cache, kv_len, block_table, max_pages, page_size, num_pages, rank, (bf16*)c_out, (bf16*)r_out, rows, status);
  VOSTI_LAUNCH_CHECK();
}

// out [tokens, heads, 128]: q [tokens, q_width] holds the queries (heads of 128 + 64) first, qr [tokens, heads, 64] their turned
// parts; kv [rows, 2 * heads * 128] keys, then the values' first terms, lo [rows, heads * 128] their second, r [rows, 64]. Every
// request's tokens are its last keys.
VOSTI_API int vosti_latent_heads(const void* q, int q_width, const void* qr, const void* kv, const void* lo, const void* r, int rows,
                                 void* out, const int* cu_q, const int* kv_len, int requests, int max_q_len, int tokens, int heads,
                                 float scale, const float* sink, const float* gate, const void* element_gate, int element_f32,
                                 int64_t element_row, unsigned* status, cudaStream_t stream) {
  VOSTI_REQUIRE(requests >= 0 && requests <= 65535 && heads > 0 && scale > 0.f, "latent_heads: bad geometry");
  VOSTI_REQUIRE(q_width % 8 == 0 && q_width >= heads * (D + ROT), "latent_heads: rows of %d elements", q_width);
  VOSTI_REQUIRE((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(qr)) % 16 == 0, "latent_heads: queries must be 16-byte aligned");
  if (requests == 0 || max_q_len <= 0 || tokens == 0) return VOSTI_OK;
  CUtensorMap mq, mqr, mkv, mlo, mr;
  VOSTI_REQUIRE(encode_tensor_map_2d(&mq, q, tokens, q_width, ROWS, 64) && encode_tensor_map_2d(&mqr, qr, tokens, heads * ROT, ROWS, 64) &&
                    encode_tensor_map_2d(&mkv, kv, rows, 2 * heads * D, KT, 64) && encode_tensor_map_2d(&mlo, lo, rows, heads * D, KT, 64) &&
                    encode_tensor_map_2d(&mr, r, rows, ROT, KT, 64), "latent_heads: cuTensorMapEncodeTiled failed");
  static const cudaError_t raised = cudaFuncSetAttribute(latent_heads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
  if (raised != cudaSuccess) {
    vosti_set_error("latent_heads: %s", cudaGetErrorString(raised));
    return (int)raised;
  }
  const int64_t row_tiles = (max_q_len + ROWS - 1) / ROWS;
  const int paired = row_tiles * heads * requests > 148;
  HeadGate g{gate, element_gate, element_f32, element_row, 0};
  g.pairs = element_gate != nullptr && !element_f32 && element_row % 2 == 0 && reinterpret_cast<uintptr_t>(element_gate) % 4 == 0;
  const int64_t ctas = heads * (paired ? (row_tiles + 1) / 2 : row_tiles);
  VOSTI_REQUIRE(ctas <= 0x7fffffff, "latent_heads: too many tiles for one launch");
  vosti_launch(latent_heads_kernel, dim3((unsigned)ctas, requests), dim3(THREADS), SMEM_BYTES, stream, mq, mqr, mkv, mlo, mr, (bf16*)out,
               cu_q, kv_len, heads, paired, scale * LOG2E, sink, g, status);
  VOSTI_LAUNCH_CHECK();
}
