// float32 matrix product on the 5th-generation tensor cores:
//   Y[t, n] = sum_k X[t, k] * W[n, k]        X, W, Y float32 (W in [out, in] layout, no bias)
// Every operand is split into three bfloat16 terms, x = h + m + l, each the upper 16 bits of what the terms before it leave
// (8 + 8 + 8 bits: nothing of a float32 is lost), and a product is the eight terms of order up to 2^-24:
// h h + (h m + m h) + (h l + m m + l h) + (m l + l m); only l l is left out, below 2^-30 of |x w| (without m l and l m a row of one
// product was 6e-8 from 64 bits instead of the 2.5e-8 of one rounding). Splitting operands this way, and
// taking the tensor core's sums out before their truncation adds up, is Ootomo and Yokota, "Recovering single
// precision accuracy from Tensor Cores while surpassing the FP32 theoretical peak performance" (2022); here h h is summed
// on the tensor core over 64 k only and then added, rounded to nearest, to a sum in registers, while the seven small products,
// 2^-7 of it, stay in an accumulator of their own to the end (over all segments, so that a row of few products is not rounded once
// a segment). Error against 64 bits (2-norm, normal operands): 1.1e-7 at K = 2,048,
// 1.4e-7 (four segments) and 2.9e-7 (one) at 4,096, 2.4e-7 at 12,288, where gemm_simt.cu's chain of multiply-adds has
// 8.1e-7, 1.1e-6 and 2.0e-6; rows of one product 2.5e-8 and of eight 2.9e-8, the chain 2.5e-8 and 5.3e-8.
//
// Features on M = 128, tokens on N; K in `segments` of whole 64s, one CTA of a cluster each, summed in their order
// through distributed shared memory. The segments are chosen from (N, K) alone, the order of the products inside a
// segment is the same in every tile width, and an output's sums never meet another's, so a row's bits never depend on the
// rows beside it (the reference chooses tiles from (N, K) only for the same reason:
// kernels/triton_kernels/matmul.py:33-73, 95-147).
//
// Operands are split times 2^16: bfloat16 ends at 2^-133, so the last terms of what lies below 2^-110 would lose bits, whatever the size of
// the output; scaled, the smallest float32 is 2^-133 and no operand loses any. The sums are exact powers of two apart and are scaled
// back at the end. Outputs that are not finite then (an infinite operand leaves inf - inf, an operand from 2^112 or a sum from 2^96 on
// overflows) go to a list that all threads work off at the end, as chains of float32 multiply-adds of the operands as they are.
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace {

constexpr int FT = 128;                  // features of a tile (MMA M)
constexpr int KCHUNK = 64;               // k that the tensor core sums before the sum is taken out
constexpr int WORKERS = 256;             // threads that load, split and sum
// Tiles of more than 128 tokens keep 96 or 128 sums a thread beside their words in flight: three warpgroups launched with
// 168 registers a thread (64,512) share them as 232 + 232 + 40.
template <int TOK> constexpr bool SPLITS_REGISTERS = TOK > 128;
template <int TOK> constexpr int THREADS = SPLITS_REGISTERS<TOK> ? WORKERS + 128 : WORKERS + 64;

// What a CTA of a tile takes of its SM. CTAs of a cluster wait for their tensor memory and for one another without a limit, so
// no more of them may be on an SM than tensor memory has columns for (512), whatever registers a build happens to give
// them: shared memory (228 KB an SM, 1 KB of it with every CTA) is padded until that many fit.
template <int TOK, int KS, int STAGES, int RAW, bool WORDS>
struct F32Tile {
  static constexpr int USED_COLS = 2 * TOK + STAGES * 3 * (KS / 2);        // the sums of 64 k, the small products, the weights' planes
  static constexpr int COLS = USED_COLS <= 256 ? 256 : 512;
  static constexpr int RINGS = STAGES * 3 * TOK * KS * 2 + (WORDS ? RAW * (FT + TOK) * KS * 4 : 0);
  static constexpr int SUMS = 2 * TOK * FT * 4 + TOK * FT;                 // a segment's, and a list of its share of the outputs, in the rings' place at the end
  static constexpr int SM_BYTES = 228 * 1024, FEWEST = SM_BYTES / (512 / COLS + 1);                        // (one CTA more does not fit)
  static constexpr int NEEDED = (RINGS > SUMS ? RINGS : SUMS) + 1024;
  static constexpr int SMEM = NEEDED > FEWEST ? NEEDED : FEWEST;
  static constexpr int COLS_AN_SM = SM_BYTES / (SMEM + 1024) * COLS;       // that its CTAs may ask for
};

__device__ __forceinline__ float4 load_cluster4(uint32_t smem_addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}
// A wait of a whole warp: one lane polls, the others meet it.
__device__ __forceinline__ bool f32_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, unsigned* status) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, abort_flag, status);
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  __syncwarp();
  return ok;
}
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory"); }
// Descriptor of a K-major tile of KS k a row: 128-byte swizzle for 64, 64-byte swizzle (groups of 8 rows 512 bytes apart) for 32.
template <int KS>
__device__ __forceinline__ uint64_t f32_desc(uint32_t addr) {
  if constexpr (KS == 64) return smem_desc_sw128(addr);
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;                // SWIZZLE_64B
  return d;
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// acc[i] += the COLS accumulator columns from `taddr` on.
template <int COLS>
__device__ __forceinline__ void add_columns(uint32_t taddr, float (&acc)[COLS]) {
  if constexpr (COLS == 32 || COLS == 64) {
#pragma unroll
    for (int c = 0; c < COLS; c += 32) {
      uint32_t r[32];
      tmem_load32(taddr + c, r);
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[c + i] += __uint_as_float(r[i]);
    }
  } else {                               // (fewer registers under way beside many sums)
    static_assert(COLS % 16 == 0, "columns");
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
      uint32_t r[16];
      tmem_load16(taddr + c, r);
#pragma unroll
      for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(r[i]);
    }
  }
}

// Four neighbouring k of a row from memory, element by element (zeros beyond k).
__device__ __forceinline__ float4 load_elements(const float* row, int kk, int k) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (kk < k) v.x = row[kk];
  if (kk + 1 < k) v.y = row[kk + 1];
  if (kk + 2 < k) v.z = row[kk + 2];
  if (kk + 3 < k) v.w = row[kk + 3];
  return v;
}
constexpr float SCALE = 65536.f, BACK = 1.f / SCALE / SCALE;
// The three terms of four values times SCALE, two values a word. A term is the upper half of what the terms before it leave (truncated: whole
// words of integer and multiply-add instructions, where a rounding conversion takes its unit several cycles), the last one is exact.
__device__ __forceinline__ void split_four(float4 x, uint32_t* h, uint32_t* m, uint32_t* l) {
  const float4 v = make_float4(x.x * SCALE, x.y * SCALE, x.z * SCALE, x.w * SCALE);
  auto upper = [](float e) { return __uint_as_float(__float_as_uint(e) & 0xffff0000u); };
  auto both = [](float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); };
  const float4 a = make_float4(v.x - upper(v.x), v.y - upper(v.y), v.z - upper(v.z), v.w - upper(v.w));
  const float4 b = make_float4(a.x - upper(a.x), a.y - upper(a.y), a.z - upper(a.z), a.w - upper(a.w));
  h[0] = both(v.x, v.y), h[1] = both(v.z, v.w);
  m[0] = both(a.x, a.y), m[1] = both(a.z, a.w);
  l[0] = both(b.x, b.y), l[1] = both(b.z, b.w);
}
// Eight columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_store8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// TOK tokens on N. One thread brings both operands' words of KS k into a ring of RAW stages by TMA (zeros beyond a matrix), eight
// warps split them, the weights into three planes in tensor memory (a thread: half a feature's k), the tokens into three in
// shared memory, and between stages take the tensor core's 64-k sums out (a thread: one feature, TOK / 2 tokens); a ninth warp
// issues the MMAs. With the weights' planes in shared memory too, every product read them again (10 KB for each MMA of 192 tokens):
// six products, us for 24,576 x 4,096, 1 / 64 / 384 rows, 152 / 283 / 570 so and 91 / 161 / 432 as it is; the eight products of
// scaled operands take 99 / 169 / 494, gemm_simt.cu 155 / 435 / 1,699. At 384 rows the tensor cores are 64 % busy, issue slots 47 %,
// shared memory 37 %. The roles share no code from where they part (their registers differ): the warps that bring and issue end after
// their last request, the eight do the rest.
// WORDS: every row starts on a whole word; otherwise the eight warps read the matrices themselves, element by element.
template <int TOK, int KS, int STAGES, int RAW, int BLOCKS, bool WORDS>
__global__ void __launch_bounds__(THREADS<TOK>, BLOCKS)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ x,
                const float* __restrict__ w, float* __restrict__ y, int rows, int n, int k, int token_tiles, int segments, unsigned* status) {
  static_assert(KS == 32 || KS == 64, "k of a ring stage");
  constexpr int ROW = KS * 2;                               // bytes of a row in a plane
  constexpr int B_PLANE = TOK * ROW, A_COLS = KS / 2;       // of a plane
  constexpr int STAGE = 3 * B_PLANE, RAW_STAGE = WORDS ? (FT + TOK) * KS * 4 : 0;
  constexpr int BW = TOK * KS / 4 / WORKERS;                // token words a thread splits per stage
  constexpr int ROWS_PER = WORKERS / (KS / 4);              // rows between a thread's words
  constexpr int COLS = TOK / 2;
  using Tile = F32Tile<TOK, KS, STAGES, RAW, WORDS>;
  constexpr int TMEM_COLS = Tile::COLS;
  static_assert(ROWS_PER % 8 == 0 && TOK * KS / 4 % WORKERS == 0 && Tile::USED_COLS <= 512 && TMEM_COLS * BLOCKS <= 512 && Tile::COLS_AN_SM <= 512, "tile");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  // [RAW] stages: the weights' [KS / 32][128 features][32] with the 128-byte swizzle, the tokens' [TOK][KS]
  uint8_t* const words = smem + STAGES * STAGE;
  __shared__ __align__(8) uint64_t raw_full[RAW], raw_empty[RAW];
  __shared__ __align__(8) uint64_t full_bar[STAGES];        // eight warps: a stage is split and stored
  __shared__ __align__(8) uint64_t empty_bar[STAGES];       // its MMAs are complete
  __shared__ __align__(8) uint64_t sum_free;                // eight warps: the 64-k sum has been taken out
  __shared__ uint32_t tmem_base_holder;
  __shared__ int again;                                     // outputs on the list
  __shared__ volatile int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int segment = blockIdx.x % segments;
  const int t0 = (blockIdx.x / segments) % token_tiles * TOK, f0 = blockIdx.x / (segments * token_tiles) * FT;
  const int chunks = (k + KCHUNK - 1) / KCHUNK;
  const int c_begin = (int)((long long)chunks * segment / segments), c_end = (int)((long long)chunks * (segment + 1) / segments);
  const int stages = (c_end - c_begin) * (KCHUNK / KS), k_begin = c_begin * KCHUNK;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    again = 0;
    for (int s = 0; s < RAW; ++s) {
      mbar_init(smem_u32(&raw_full[s]), 1);
      mbar_init(smem_u32(&raw_empty[s]), WORKERS / 32);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), WORKERS / 32);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&sum_free), WORKERS / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(&tmem_base_holder), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();               // (after this CTA's tensor memory is its own)
  const uint32_t tmem_sum = tmem_base_holder, tmem_small = tmem_sum + TOK, tmem_a = tmem_small + TOK;

  if (warp >= WORKERS / 32) {
    if constexpr (SPLITS_REGISTERS<TOK>) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == WORKERS / 32 + 1 && lane == 0 && WORDS) {
      // the weights of the first stages do not depend on the kernel before this one
      auto bring_w = [&](int st) {
        const int s = st % RAW;
        mbar_expect_tx(smem_u32(&raw_full[s]), (uint32_t)RAW_STAGE);
        for (int p = 0; p < KS / 32; ++p)
          tma_load_2d(smem_u32(words + s * RAW_STAGE + p * FT * 128), &map_w, k_begin + st * KS + p * 32, f0, smem_u32(&raw_full[s]));
      };
      auto bring_x = [&](int st) {
        const int s = st % RAW;
        tma_load_2d(smem_u32(words + s * RAW_STAGE + FT * KS * 4), &map_x, k_begin + st * KS, t0, smem_u32(&raw_full[s]));
      };
      const int first = stages < RAW ? stages : RAW;
      for (int st = 0; st < first; ++st) bring_w(st);
      pdl_wait();
      for (int st = 0; st < first; ++st) bring_x(st);
      for (int st = first; st < stages; ++st) {
        if (!mbar_wait(smem_u32(&raw_empty[st % RAW]), (st / RAW - 1) & 1, &abort_flag, status)) break;
        bring_w(st);
        bring_x(st);
      }
    }
    if (warp == WORKERS / 32) {
      constexpr uint32_t idesc = umma_instr_desc(FT, TOK, false);
      bool ok = true;
      auto arrived = [&](uint64_t* bar, uint32_t parity) {
        return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, &abort_flag, status)) != 0;
      };
      for (int st = 0; st < stages && ok; ++st) {
        const int s = st % STAGES;
        ok = arrived(&full_bar[s], (st / STAGES) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ah = tmem_a + s * 3 * A_COLS, am = ah + A_COLS, al = am + A_COLS, bb = smem_u32(smem + s * STAGE);
        const uint64_t bh = f32_desc<KS>(bb), bm = f32_desc<KS>(bb + B_PLANE), bl = f32_desc<KS>(bb + 2 * B_PLANE);
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < KS / 16; ++q) {
            umma_bf16_ts(tmem_small, al + 8 * q, bm + 2 * q, idesc, st > 0 || q > 0);
            umma_bf16_ts(tmem_small, am + 8 * q, bl + 2 * q, idesc, 1u);
            umma_bf16_ts(tmem_small, al + 8 * q, bh + 2 * q, idesc, 1u);
            umma_bf16_ts(tmem_small, am + 8 * q, bm + 2 * q, idesc, 1u);
            umma_bf16_ts(tmem_small, ah + 8 * q, bl + 2 * q, idesc, 1u);
            umma_bf16_ts(tmem_small, am + 8 * q, bh + 2 * q, idesc, 1u);
            umma_bf16_ts(tmem_small, ah + 8 * q, bm + 2 * q, idesc, 1u);
          }
        }
        __syncwarp();
        const int chunk = st / (KCHUNK / KS), part = st % (KCHUNK / KS);
        if (part == 0 && chunk > 0) {
          ok = arrived(&sum_free, (chunk - 1) & 1);
          if (!ok) break;
          tc_fence_after();
        }
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < KS / 16; ++q) umma_bf16_ts(tmem_sum, ah + 8 * q, bh + 2 * q, idesc, part > 0 || q > 0);
          umma_commit(smem_u32(&empty_bar[s]));
        }
        __syncwarp();
      }
    }
    return;
  }

  if constexpr (SPLITS_REGISTERS<TOK>) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
  pdl_wait();
  float acc[COLS];
#pragma unroll
  for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
  const int quarter = warp & 3, half = warp >> 2;
  const uint32_t my_columns = ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * COLS);
  // weights: half of feature `quarter * 32 + lane`'s k, whose words lie at its place in the swizzle pattern
  const int feature = quarter * 32 + lane;
  const uint32_t my_a = tmem_a + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * (A_COLS / 2));
  // tokens:
  const int my_row = threadIdx.x / (KS / 4), my_k = threadIdx.x % (KS / 4) * 4;
  const int rows_here = rows - t0;
  // (a thread's rows are a multiple of 8 apart: one place in the swizzle pattern for all of them)
  const int place = my_row * ROW + (((my_k >> 3) ^ (KS == 64 ? my_row & 7 : (my_row >> 1) & 3)) << 4) + (my_k & 4) * 2;
  bool ok = true;
  for (int st = 0; st < stages + STAGES; ++st) {
    const int s = st % STAGES;
    if (st >= STAGES) {
      // the stage that held this slot is complete: with it, at a chunk's end, the sum over 64 k
      ok = ok && f32_wait(smem_u32(&empty_bar[s]), (st / STAGES - 1) & 1, &abort_flag, status);
      if (ok && (st - STAGES) % (KCHUNK / KS) == KCHUNK / KS - 1) {
        tc_fence_after();
        add_columns<COLS>(tmem_sum + my_columns, acc);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sum_free));
      }
    }
    if (!ok || st >= stages) continue;
    const uint8_t* const raw = words + st % RAW * RAW_STAGE;
    if (WORDS) {
      ok = f32_wait(smem_u32(&raw_full[st % RAW]), (st / RAW) & 1, &abort_flag, status);
      if (!ok) continue;
    }
    if (st >= STAGES) tc_fence_after();                    // (the MMAs that read the slot's planes)
#pragma unroll
    for (int g = 0; g < KS / 32; ++g) {
      uint32_t h[8], m[8], l[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int kk = half * (KS / 2) + g * 16 + i * 4;
        const float4 v = WORDS ? *reinterpret_cast<const float4*>(raw + (kk / 32 * FT + feature) * 128 + (((kk % 32 >> 2) ^ (feature & 7)) << 4))
                               : load_elements(w + (int64_t)min(f0 + feature, n - 1) * k, k_begin + st * KS + kk, k);
        split_four(v, h + 2 * i, m + 2 * i, l + 2 * i);
      }
      const uint32_t at = my_a + s * 3 * A_COLS + g * 8;
      tmem_store8(at, h);
      tmem_store8(at + A_COLS, m);
      tmem_store8(at + 2 * A_COLS, l);
    }
#pragma unroll
    for (int i = 0; i < BW; ++i) {
      const int r = my_row + i * ROWS_PER;
      // (columns of rows that are not there are never stored, and touch no other column)
      if (TOK <= 64 && r >= rows_here) continue;
      const float4 v = WORDS ? *reinterpret_cast<const float4*>(raw + FT * KS * 4 + (r * KS + my_k) * 4)
                             : load_elements(x + (int64_t)min(t0 + r, rows - 1) * k, k_begin + st * KS + my_k, k);
      uint2 h, m, l;
      split_four(v, &h.x, &m.x, &l.x);
      uint8_t* const at = smem + s * STAGE + i * ROWS_PER * ROW + place;
      *reinterpret_cast<uint2*>(at) = h;
      *reinterpret_cast<uint2*>(at + B_PLANE) = m;
      *reinterpret_cast<uint2*>(at + 2 * B_PLANE) = l;
    }
    tmem_wait_stores();
    tc_fence_before();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(smem_u32(&full_bar[s]));
      if (WORDS) mbar_arrive(smem_u32(&raw_empty[st % RAW]));
    }
  }
  tc_fence_after();
  if (ok && segments == 1) add_columns<COLS>(tmem_small + my_columns, acc);

  uint16_t* const list = reinterpret_cast<uint16_t*>(segments == 1 ? smem : smem + 2 * TOK * FT * 4);     // outputs to be taken again
  auto store = [&](int t, int f, float v) {
    if (t0 + t >= rows || f0 + f >= n) return;
    if (fabsf(v) <= 3.402823466e+38f) y[(int64_t)(t0 + t) * n + f0 + f] = v * BACK;
    else list[atomicAdd(&again, 1)] = (uint16_t)(t * FT + f);
  };
  if (segments == 1) {
    workers_sync();                                        // (all have split their last words: the rings' place is free)
#pragma unroll
    for (int i = 0; i < COLS; ++i) store(half * COLS + i, feature, acc[i]);
  } else {
    // every MMA that read the ring is complete: its place takes the sums, then the small products
    float* const part = reinterpret_cast<float*>(smem);
    float* const mine_at = part + half * COLS * FT + feature;
#pragma unroll
    for (int i = 0; i < COLS; ++i) {
      mine_at[i * FT] = acc[i];
      acc[i] = 0.f;
    }
    if (ok) add_columns<COLS>(tmem_small + my_columns, acc);
#pragma unroll
    for (int i = 0; i < COLS; ++i) mine_at[(TOK + i) * FT] = acc[i];
    cluster_sync_all();
    const int mine = (int)cluster_rank();              // = segment
    const int lo = TOK * mine / segments, hi = TOK * (mine + 1) / segments;
    for (int word = threadIdx.x; word < (hi - lo) * (FT / 4); word += WORKERS) {
      const int t = lo + word / (FT / 4), f = word % (FT / 4) * 4;
      if (t0 + t >= rows) break;
      const uint32_t at = smem_u32(&part[t * FT + f]), small_at = smem_u32(&part[(TOK + t) * FT + f]);
      float4 v = load_cluster4(at, 0), low = load_cluster4(small_at, 0);
      for (int r = 1; r < segments; ++r) {
        const float4 u = load_cluster4(at, r), e = load_cluster4(small_at, r);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        low.x += e.x; low.y += e.y; low.z += e.z; low.w += e.w;
      }
      store(t, f, v.x + low.x);
      store(t, f + 1, v.y + low.y);
      store(t, f + 2, v.z + low.z);
      store(t, f + 3, v.w + low.w);
    }
  }
  tc_fence_before();
  workers_sync();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    workers_sync();
  }
  for (int i = threadIdx.x; i < again; i += WORKERS) {
    const int t = t0 + list[i] / FT, f = f0 + list[i] % FT;
    if (t >= rows || f >= n) continue;                     // (the list's place after a wait that gave up)
    const float *xr = x + (int64_t)t * k, *wr = w + (int64_t)f * k;
    float v = 0.f;
#pragma unroll 8
    for (int kk = 0; kk < k; ++kk) v = fmaf(xr[kk], wr[kk], v);
    y[(int64_t)t * n + f] = v;
  }
  if (segments > 1) cluster_sync_all();                     // nobody reads this CTA's sums after this
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_sum, TMEM_COLS);
  }
}

// K segments: from (n, k) alone, so that few rows still start enough CTAs.
int f32_segments(int n, int k) {
  const int tiles = (n + FT - 1) / FT, chunks = (k + KCHUNK - 1) / KCHUNK;
  int s = 1;
  while (s < 8 && tiles * s * 2 <= 192 && chunks >= 8 * s) s *= 2;
  return s;
}

// Map of a row-major [rows, k] float32 matrix (k a multiple of 4, 16-byte aligned), boxes of box_rows x box_k.
bool f32_map(CUtensorMap* map, const float* base, int64_t rows, int k, int box_rows, int box_k, CUtensorMapSwizzle swizzle) {
  VostiEncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)k * 4};
  const cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TOK, int KS, int STAGES, int RAW, int BLOCKS, bool WORDS>
int launch_f32(const float* x, const float* w, float* y, int rows, int n, int k, unsigned* status, cudaStream_t stream) {
  constexpr int SMEM = F32Tile<TOK, KS, STAGES, RAW, WORDS>::SMEM;
  auto kernel = gemm_f32_kernel<TOK, KS, STAGES, RAW, BLOCKS, WORDS>;
  static const cudaError_t raised = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (raised != cudaSuccess) {
    vosti_set_error("gemm_f32: %s", cudaGetErrorString(raised));
    return (int)raised;
  }
  CUtensorMap mx = {}, mw = {};
  VOSTI_REQUIRE(!WORDS || (f32_map(&mx, x, rows, k, TOK, KS, CU_TENSOR_MAP_SWIZZLE_NONE) && f32_map(&mw, w, n, k, FT, 32, CU_TENSOR_MAP_SWIZZLE_128B)),
                "gemm_f32: cuTensorMapEncodeTiled failed");
  const int segments = f32_segments(n, k), token_tiles = (rows + TOK - 1) / TOK;
  const int64_t ctas = (int64_t)((n + FT - 1) / FT) * token_tiles * segments;
  VOSTI_REQUIRE(ctas <= 0x7fffffff, "gemm_f32: too many tiles for one launch");
  const cudaError_t e = vosti_launch_clusters(kernel, dim3((unsigned)ctas), dim3(THREADS<TOK>), (unsigned)segments, SMEM, stream, mx, mw, x, w,
                                              y, rows, n, k, token_tiles, segments, status);
  if (e != cudaSuccess) {
    vosti_set_error("gemm_f32: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return VOSTI_OK;
}

template <int TOK, int KS, int STAGES, int RAW>
constexpr int f32_cols_an_sm() {
  const int words = F32Tile<TOK, KS, STAGES, RAW, true>::COLS_AN_SM, elements = F32Tile<TOK, KS, STAGES, RAW, false>::COLS_AN_SM;
  return words > elements ? words : elements;
}

}  // namespace

// Tensor memory columns that the CTAs of a tile (0 .. 5, -1 beyond) may ask for on one SM.
VOSTI_API int vosti_gemm_f32_columns_an_sm(int tile) {
  constexpr int of[] = {f32_cols_an_sm<32, 64, 2, 3>(), f32_cols_an_sm<32, 64, 2, 2>(), f32_cols_an_sm<64, 64, 2, 2>(),
                        f32_cols_an_sm<64, 32, 2, 3>(), f32_cols_an_sm<128, 64, 2, 2>(), f32_cols_an_sm<192, 32, 2, 2>()};
  return tile >= 0 && tile < (int)(sizeof(of) / sizeof(of[0])) ? of[tile] : -1;
}

// Whether a float32 [n, k] weight is this kernel's (a rule of the sizes only, so that a row's bits stay its own): where one row is no slower
// than gemm_simt.cu's chain of multiply-adds; with more rows it is faster from 8 to 16 on everywhere. us, here / there, one row: 1,024 x 1,024
// 7.7 / 6.6, 3,072 x 1,024 9.2 / 7.4, 4,096 x 1,024 9.9 / 9.8, 8,192 x 1,024 13.6 / 13.9, 2,048 x 1,920 12.0 / 11.2, 4,096 x 1,536 12.0 / 13.2,
// 16 x 2,048 7.6 / 10.2, 2,048 x 2,048 10.5 / 11.3, 2,048 x 2,304 11.8 / 12.2. Rows that do not start on whole words are read element
// by element: 4,096 x 4,098 60 / 39.
VOSTI_API int vosti_gemm_f32_supported(int n, int k) { return n >= 16 && k % 4 == 0 && (k >= 2048 || (k >= 1024 && n >= 4096)); }

// x: [rows, k]; w: [n, k]; y: [rows, n], all float32.
VOSTI_API int vosti_gemm_f32(const float* x, const float* w, float* y, int rows, int n, int k, unsigned* status, cudaStream_t stream) {
  VOSTI_REQUIRE(rows >= 0 && n > 0 && k > 0, "gemm_f32: bad sizes rows=%d n=%d k=%d", rows, n, k);
  if (rows == 0) return VOSTI_OK;
  // every row starts on a whole word
  const bool wide = k % 4 == 0 && (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) % 16 == 0;
#define VOSTI_F32(TOK, KS, STAGES, RAW, BLOCKS) \
  return wide ? launch_f32<TOK, KS, STAGES, RAW, BLOCKS, true>(x, w, y, rows, n, k, status, stream) \
              : launch_f32<TOK, KS, STAGES, RAW, BLOCKS, false>(x, w, y, rows, n, k, status, stream)
  const int tiles = (n + FT - 1) / FT, segments = f32_segments(n, k);
  auto ctas = [&](int tok) { return (int64_t)tiles * segments * ((rows + tok - 1) / tok); };
  // Clusters of up to four CTAs find some 140 SMs at one CTA each. Where these take them all at once, a deeper ring of whole 64s is the
  // fastest (us, 4,096 x 12,288, 1 row: 54, two stages 73, stages of 32 k 108; 64 rows: 77 and 128); with more CTAs, or eight a
  // cluster, two of them an SM are (24,576 x 4,096, 1 row: 101 and 136, 64 rows: 176 and 194; 2,048 x 2,048: 11 and 17, 19 and 27).
  const bool one_round = segments <= 4 && ctas(rows) <= 140;
  if (rows <= 32 && one_round) VOSTI_F32(32, 64, 2, 3, 1);
  if (rows <= 32) VOSTI_F32(32, 64, 2, 2, 2);
  if (rows <= 64 && one_round) VOSTI_F32(64, 64, 2, 2, 1);
  if (rows <= 64) VOSTI_F32(64, 32, 2, 3, 2);
  // A tile of 192 tokens takes about 1.4 times as long as one of 128: the fewer rounds of CTAs decide (us, 384 rows: 24,576 x 4,096 546
  // and 486, 6,144 x 4,096 164 and 186, 4,096 x 4,096 109 and 113).
  const int at_once = segments > 1 ? 140 : 148;
  if (10 * ((ctas(128) + at_once - 1) / at_once) <= 14 * ((ctas(192) + at_once - 1) / at_once)) VOSTI_F32(128, 64, 2, 2, 1);
  VOSTI_F32(192, 32, 2, 2, 1);
#undef VOSTI_F32
}
