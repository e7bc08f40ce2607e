// float32 matrix product on the 5th-generation tensor cores:
//   Y[t, n] = sum_k X[row(t), k] * W[n, k]        X, W, Y float32 (W in [out, in] layout, no bias)
// Every operand is split into three bfloat16 terms, x = h + m + l, each the rounding of what the terms before it leave
// (8 + 8 + 8 bits: nothing of a float32 is lost), and a product is the six terms of order up to 2^-16:
// h h + (h m + m h) + (h l + m m + l h); what is left out is below 2^-25 of |x w|. Splitting operands this way, and taking
// the tensor core's sums out before their truncation adds up, is Ootomo and Yokota, "Recovering single
// precision accuracy from Tensor Cores while surpassing the FP32 theoretical peak performance" (2022); here h h is summed
// on the tensor core over 64 k only and then added, rounded to nearest, to a sum in registers, while the five small products,
// 2^-8 of it, stay in an accumulator of their own to the end. Error against 64 bits (2-norm, normal operands): 1.1e-7
// at K = 4,096 and 1.3e-7 at 12,288, where gemm_simt.cu's chain of multiply-adds has 1.2e-6 and 2.0e-6.
//
// Features on M = 128, tokens on N; K in `segments` of whole 64s, one CTA of a cluster each, summed in their order
// through distributed shared memory. The segments are chosen from (N, K) alone, the order of the products inside a
// segment is the same in every tile width, and an output's sums never meet another's, so a row's bits never depend on the
// rows beside it (the reference chooses tiles from (N, K) only for the same reason:
// kernels/triton_kernels/matmul.py:33-73, 95-147).
//
// An operand that is infinite, not a number or rounds to infinity in 16 bits makes its outputs non-finite here, and terms of
// operands near the smallest normal number lose their low bits; outputs that are not finite, or so small that this could show
// (below 2^-80 and not zero), are taken again as a chain of float32 multiply-adds.
#include "tcgen05.cuh"

namespace {

constexpr int FT = 128;                  // features of a tile (MMA M)
constexpr int KCHUNK = 64;               // k that the tensor core sums before the sum is taken out
constexpr int WORKERS = 256;             // threads that load, split and sum
// Tiles of more than 128 tokens keep 96 or 128 sums a thread beside their words in flight: three warpgroups launched with
// 168 registers a thread (64,512) share them as 232 + 232 + 40.
template <int TOK> constexpr bool SPLITS_REGISTERS = TOK > 128;
template <int TOK> constexpr int THREADS = SPLITS_REGISTERS<TOK> ? WORKERS + 128 : WORKERS + 32;

__device__ __forceinline__ uint32_t f32_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void f32_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 load_cluster4(uint32_t smem_addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
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

// Four neighbouring k of a row (zeros beyond k, or of a row that is not there).
__device__ __forceinline__ float4 load_word(const float* matrix, int row, int kk, int k, bool wide) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row < 0 || kk >= k) return v;
  const float* p = matrix + (int64_t)row * k + kk;
  if (wide) return *reinterpret_cast<const float4*>(p);
  v.x = p[0];
  if (kk + 1 < k) v.y = p[1];
  if (kk + 2 < k) v.z = p[2];
  if (kk + 3 < k) v.w = p[3];
  return v;
}
// The three terms of four values to their places in three planes of `plane` bytes.
__device__ __forceinline__ void store_split(uint8_t* at, int plane, float4 v) {
  const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
  const float2 a = __bfloat1622float2(h0), b = __bfloat1622float2(h1);
  v.x -= a.x; v.y -= a.y; v.z -= b.x; v.w -= b.y;
  const __nv_bfloat162 m0 = __floats2bfloat162_rn(v.x, v.y), m1 = __floats2bfloat162_rn(v.z, v.w);
  const float2 c = __bfloat1622float2(m0), d = __bfloat1622float2(m1);
  v.x -= c.x; v.y -= c.y; v.z -= d.x; v.w -= d.y;
  const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x, v.y), l1 = __floats2bfloat162_rn(v.z, v.w);
  auto put = [&](uint8_t* p, const __nv_bfloat162& lo, const __nv_bfloat162& hi) {
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  };
  put(at, h0, h1);
  put(at + plane, m0, m1);
  put(at + 2 * plane, l0, l1);
}

// TOK tokens on N. Eight warps load words of both operands into registers (AHEAD stages ahead), split them into the three
// planes of a ring stage of KS k, and between stages take the tensor core's 64-k sums out (thread: one feature, TOK / 2 tokens);
// one lane of the ninth warp issues the MMAs. The two roles share no code from where they part (their registers differ):
// the ninth warp ends after its last commit, the eight do the rest. The fence between the warps' stores and the MMAs that read
// them (generic to async proxy) is the issuing lane's, after its wait: in the eight warps it would also wait for
// the words of the next stages that are under way.
template <int TOK, int KS, int STAGES, int AHEAD, int BLOCKS>
__global__ void __launch_bounds__(THREADS<TOK>, BLOCKS)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, const int* __restrict__ row_index,
                int rows, int x_rows, int n, int k, int token_tiles, int segments, int wide, unsigned* status) {
  static_assert(KS == 32 || KS == 64, "k of a ring stage");
  constexpr int ROW = KS * 2;                               // bytes of a row in a plane
  constexpr int A_PLANE = FT * ROW, B_PLANE = TOK * ROW;
  constexpr int STAGE = 3 * (A_PLANE + B_PLANE);
  constexpr int AW = FT * KS / 4 / WORKERS, BW = TOK * KS / 4 / WORKERS;     // words a thread brings per stage
  constexpr int ROWS_PER = WORKERS / (KS / 4);              // rows between a thread's words
  constexpr int COLS = TOK / 2;
  constexpr int TMEM_COLS = 2 * TOK <= 64 ? 64 : 2 * TOK <= 128 ? 128 : 2 * TOK <= 256 ? 256 : 512;
  static_assert(TOK * KS / 4 % WORKERS == 0 && STAGES * STAGE >= TOK * FT * 4, "tile");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES];        // eight warps: a stage is split and stored
  __shared__ __align__(8) uint64_t empty_bar[STAGES];       // its MMAs are complete
  __shared__ __align__(8) uint64_t sum_free;                // eight warps: the 64-k sum has been taken out
  __shared__ uint32_t tmem_base_holder;
  __shared__ volatile int abort_flag;
  __shared__ int source[TOK];                               // rows of x; -1: zeros, for an index out of range; -2: none

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int segment = blockIdx.x % segments;
  const int t0 = (blockIdx.x / segments) % token_tiles * TOK, f0 = blockIdx.x / (segments * token_tiles) * FT;
  const int chunks = (k + KCHUNK - 1) / KCHUNK;
  const int c_begin = (int)((long long)chunks * segment / segments), c_end = (int)((long long)chunks * (segment + 1) / segments);
  const int stages = (c_end - c_begin) * (KCHUNK / KS), k_begin = c_begin * KCHUNK;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), WORKERS / 32);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&sum_free), WORKERS / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(&tmem_base_holder), TMEM_COLS);
  // the weights do not depend on the kernel before this one
  const int my_row = threadIdx.x / (KS / 4), my_k = threadIdx.x % (KS / 4) * 4;
  float4 a[AHEAD][AW], b[AHEAD][BW];
  auto fetch_a = [&](float4 (&to)[AW], int stage) {
#pragma unroll
    for (int i = 0; i < AW; ++i) {
      const int f = f0 + my_row + i * ROWS_PER;
      to[i] = load_word(w, f < n ? f : -1, k_begin + stage * KS + my_k, k, wide);
    }
  };
  auto fetch_b = [&](float4 (&to)[BW], int stage) {
#pragma unroll
    for (int i = 0; i < BW; ++i) to[i] = load_word(x, source[my_row + i * ROWS_PER], k_begin + stage * KS + my_k, k, wide);
  };
  if (warp < WORKERS / 32) {
#pragma unroll
    for (int p = 0; p < AHEAD; ++p)
      if (p < stages) fetch_a(a[p], p);
  }
  pdl_wait();
  for (int t = threadIdx.x; t < TOK; t += THREADS<TOK>) {
    int from = -2;
    if (t0 + t < rows) {
      from = row_index ? row_index[t0 + t] : t0 + t;
      if (from < 0 || from >= x_rows) {
        raise_fault(status, VOSTI_FAULT_ROW_RANGE);
        from = -1;
      }
    }
    source[t] = from;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();               // (after this CTA's tensor memory is its own)
  const uint32_t tmem_sum = tmem_base_holder, tmem_small = tmem_sum + TOK;

  if (warp >= WORKERS / 32) {
    if constexpr (SPLITS_REGISTERS<TOK>) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == WORKERS / 32 && lane == 0) {
      constexpr uint32_t idesc = umma_instr_desc(FT, TOK, false);
      bool ok = true;
      for (int st = 0; st < stages && ok; ++st) {
        const int s = st % STAGES;
        ok = mbar_wait(smem_u32(&full_bar[s]), (st / STAGES) & 1, &abort_flag, status);
        if (!ok) break;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_after();
        const uint32_t base = smem_u32(smem + s * STAGE);
        const uint64_t ah = f32_desc<KS>(base), am = f32_desc<KS>(base + A_PLANE), al = f32_desc<KS>(base + 2 * A_PLANE);
        const uint32_t bb = base + 3 * A_PLANE;
        const uint64_t bh = f32_desc<KS>(bb), bm = f32_desc<KS>(bb + B_PLANE), bl = f32_desc<KS>(bb + 2 * B_PLANE);
#pragma unroll
        for (int q = 0; q < KS / 16; ++q) {
          umma_bf16(tmem_small, al + 2 * q, bh + 2 * q, idesc, st > 0 || q > 0);
          umma_bf16(tmem_small, am + 2 * q, bm + 2 * q, idesc, 1u);
          umma_bf16(tmem_small, ah + 2 * q, bl + 2 * q, idesc, 1u);
          umma_bf16(tmem_small, am + 2 * q, bh + 2 * q, idesc, 1u);
          umma_bf16(tmem_small, ah + 2 * q, bm + 2 * q, idesc, 1u);
        }
        const int chunk = st / (KCHUNK / KS), part = st % (KCHUNK / KS);
        if (part == 0 && chunk > 0) {
          ok = mbar_wait(smem_u32(&sum_free), (chunk - 1) & 1, &abort_flag, status);
          if (!ok) break;
          tc_fence_after();
        }
#pragma unroll
        for (int q = 0; q < KS / 16; ++q) umma_bf16(tmem_sum, ah + 2 * q, bh + 2 * q, idesc, part > 0 || q > 0);
        umma_commit(smem_u32(&empty_bar[s]));
      }
    }
    return;
  }

  if constexpr (SPLITS_REGISTERS<TOK>) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
  float acc[COLS];
#pragma unroll
  for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
  const int quarter = warp & 3, half = warp >> 2;
  const uint32_t my_columns = ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * COLS);
#pragma unroll
  for (int p = 0; p < AHEAD; ++p)
    if (p < stages) fetch_b(b[p], p);
  bool ok = true;
  auto swizzle = [](int r) { return KS == 64 ? r & 7 : (r >> 1) & 3; };
  auto step = [&](float4 (&aw)[AW], float4 (&bw)[BW], int st) {
    const int s = st % STAGES;
    if (st >= STAGES) {
      // the stage that held this slot is complete: with it, at a chunk's end, the sum over 64 k
      ok = ok && mbar_wait_warp(smem_u32(&empty_bar[s]), (st / STAGES - 1) & 1, &abort_flag, status);
      if (ok && (st - STAGES) % (KCHUNK / KS) == KCHUNK / KS - 1) {
        tc_fence_after();
        add_columns<COLS>(tmem_sum + my_columns, acc);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sum_free));
      }
    }
    if (!ok || st >= stages) return;
    uint8_t* const base = smem + s * STAGE;
#pragma unroll
    for (int i = 0; i < AW; ++i) {
      const int r = my_row + i * ROWS_PER;
      store_split(base + r * ROW + (((my_k >> 3) ^ swizzle(r)) << 4) + (my_k & 4) * 2, A_PLANE, aw[i]);
    }
#pragma unroll
    for (int i = 0; i < BW; ++i) {
      const int r = my_row + i * ROWS_PER;
      // (columns of rows that are not there are never stored, and touch no other column)
      if (TOK <= 64 && source[r] == -2) continue;
      store_split(base + 3 * A_PLANE + r * ROW + (((my_k >> 3) ^ swizzle(r)) << 4) + (my_k & 4) * 2, B_PLANE, bw[i]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&full_bar[s]));
    if (st + AHEAD < stages) {
      fetch_a(aw, st + AHEAD);
      fetch_b(bw, st + AHEAD);
    }
  };
  for (int st = 0; st < stages + STAGES; st += AHEAD) {
#pragma unroll
    for (int p = 0; p < AHEAD; ++p)
      if (st + p < stages + STAGES) step(a[p], b[p], st + p);
  }
  if (ok) {
    tc_fence_after();
    add_columns<COLS>(tmem_small + my_columns, acc);
    tc_fence_before();
  }

  auto store = [&](int t, int f, float v) {
    if (t0 + t >= rows || f0 + f >= n) return;
    if (!(fabsf(v) <= 3.402823466e+38f) || (fabsf(v) < 8.2718061e-25f && v != 0.f)) {       // 2^-80
      v = 0.f;
      const int from = source[t];
      const float *xr = x + (int64_t)(from < 0 ? 0 : from) * k, *wr = w + (int64_t)(f0 + f) * k;
      for (int kk = 0; kk < k && v == v; ++kk) v = fmaf(from < 0 ? 0.f : xr[kk], wr[kk], v);
    }
    y[(int64_t)(t0 + t) * n + f0 + f] = v;
  };
  if (segments == 1) {
#pragma unroll
    for (int i = 0; i < COLS; ++i) store(half * COLS + i, quarter * 32 + lane, acc[i]);
  } else {
    // every MMA that read the ring is complete
    float* const part = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int i = 0; i < COLS; ++i) part[(half * COLS + i) * FT + quarter * 32 + lane] = acc[i];
    f32_cluster_sync();
    const int mine = (int)f32_cluster_rank();              // = segment
    const int lo = TOK * mine / segments, hi = TOK * (mine + 1) / segments;
    for (int word = threadIdx.x; word < (hi - lo) * (FT / 4); word += WORKERS) {
      const int t = lo + word / (FT / 4), f = word % (FT / 4) * 4;
      if (t0 + t >= rows) break;
      const uint32_t at = smem_u32(&part[t * FT + f]);
      float4 v = load_cluster4(at, 0);
      for (int r = 1; r < segments; ++r) {
        const float4 u = load_cluster4(at, r);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
      }
      store(t, f, v.x);
      store(t, f + 1, v.y);
      store(t, f + 2, v.z);
      store(t, f + 3, v.w);
    }
  }
  tc_fence_before();
  workers_sync();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    workers_sync();
  }
  if (segments > 1) f32_cluster_sync();                     // nobody reads this CTA's sums after this
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

template <int TOK, int KS, int STAGES, int AHEAD, int BLOCKS>
int launch_f32(const float* x, const float* w, float* y, const int* row_index, int rows, int x_rows, int n, int k, int wide,
               unsigned* status, cudaStream_t stream) {
  constexpr int SMEM = STAGES * 3 * (FT + TOK) * KS * 2 + 1024;
  auto kernel = gemm_f32_kernel<TOK, KS, STAGES, AHEAD, BLOCKS>;
  static const cudaError_t raised = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (raised != cudaSuccess) {
    vosti_set_error("gemm_f32: %s", cudaGetErrorString(raised));
    return (int)raised;
  }
  const int segments = f32_segments(n, k), token_tiles = (rows + TOK - 1) / TOK;
  const int64_t ctas = (int64_t)((n + FT - 1) / FT) * token_tiles * segments;
  VOSTI_REQUIRE(ctas <= 0x7fffffff, "gemm_f32: too many tiles for one launch");
  const cudaError_t e = vosti_launch_clusters(kernel, dim3((unsigned)ctas), dim3(THREADS<TOK>), (unsigned)segments, SMEM, stream, x, w, y,
                                              row_index, rows, x_rows, n, k, token_tiles, segments, wide, status);
  if (e != cudaSuccess) {
    vosti_set_error("gemm_f32: %s", cudaGetErrorString(e));
    return (int)e;
  }
  return VOSTI_OK;
}

}  // namespace

// Whether the kernel takes a float32 [n, k] weight (a rule of the sizes only).
VOSTI_API int vosti_gemm_f32_supported(int n, int k) { return n >= 16 && k >= 128; }

// x: [x_rows, k]; w: [n, k]; y: [rows, n], all float32. With row_index (int32[rows]) row t is x[row_index[t]].
VOSTI_API int vosti_gemm_f32(const float* x, const float* w, float* y, const int* row_index, int rows, int x_rows, int n, int k,
                             unsigned* status, cudaStream_t stream) {
  VOSTI_REQUIRE(rows >= 0 && x_rows >= 0 && vosti_gemm_f32_supported(n, k), "gemm_f32: bad sizes rows=%d n=%d k=%d", rows, n, k);
  VOSTI_REQUIRE(row_index != nullptr || rows == x_rows, "gemm_f32: rows != x_rows without a row index");
  if (rows == 0) return VOSTI_OK;
  const int wide = k % 4 == 0 && (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) % 16 == 0;
#define VOSTI_F32(TOK, KS, STAGES, AHEAD, BLOCKS) \
  return launch_f32<TOK, KS, STAGES, AHEAD, BLOCKS>(x, w, y, row_index, rows, x_rows, n, k, wide, status, stream)
  const int by256 = (rows + 255) / 256 * 256, by192 = (rows + 191) / 192 * 192;
  if (rows <= 32) VOSTI_F32(32, 32, 3, 2, 2);
  if (rows <= 64) VOSTI_F32(64, 32, 3, 1, 2);
  if (rows <= 128) VOSTI_F32(128, 32, 4, 1, 1);
  if (by192 < by256) VOSTI_F32(192, 32, 3, 1, 1);
  VOSTI_F32(256, 32, 3, 1, 1);
#undef VOSTI_F32
}
