// Plain matrix product on the CUDA cores with true float32 arithmetic:
//   Y[t, n] = sum_k X[row(t), k] * W[n, k]        (W in [out, in] layout, no bias)
// It is the float32 product of weights that gemm_f32.cu does not take (`vosti_gemm_f32_supported`) and the fallback of the bfloat16 path for
// operand types or sizes the tensor-core kernel refuses. Each output is one thread's
// sequential fused multiply-add chain over k = 0..K-1, so a row's value never depends
// on the other rows of the launch (the reference's matmul has the same property by
// choosing tiles from (N, K) only: kernels/triton_kernels/matmul.py:33-73, 95-147). The tile itself is
// chosen by how many outputs there are (see `launch`).
#include "common.cuh"

namespace {

// Four neighbouring k of a row as float32; beyond k, or of a row that is not there (-1), zeros.
template <typename T>
__device__ __forceinline__ float4 load4_of(const T* matrix, int r, int kk, int k, bool wide) {
  if (wide || sizeof(T) == 4) {
    if (r < 0 || kk >= k) return make_float4(0.f, 0.f, 0.f, 0.f);
    const T* row = matrix + (int64_t)r * k;
    if (wide) return load_four(row + kk);
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = kk + i < k ? to_f32(row[kk + i]) : 0.f;
    return make_float4(v[0], v[1], v[2], v[3]);
  }
  // Single bfloat16 elements: no branch between the four loads (those that are not wanted read the row's last one, or
  // row 0's), since each is converted at once and would wait for the one before it: 384 x 4,096 x 4,097 478 us
  // instead of 430 in tiles of 64 x 64, 65 rows 338 instead of 199.
  const T* const row = matrix + (int64_t)(r < 0 ? 0 : r) * k;
  T raw[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) raw[i] = row[kk + i < k ? kk + i : k - 1];
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = r >= 0 && kk + i < k ? to_f32(raw[i]) : 0.f;
  return make_float4(v[0], v[1], v[2], v[3]);
}

// The words of four k that a thread brings of a block's BM rows of x and BN rows of w, BK of k at a time:
// fetched into registers while the BK before them are multiplied.
template <typename TX, typename TW, int BM, int BN, int BK, int THREADS>
struct TileLoads {
  static constexpr int WORDS = BK / 4;
  static constexpr int XL = (BM * WORDS + THREADS - 1) / THREADS, WL = (BN * WORDS + THREADS - 1) / THREADS;
  int xrow[XL], wrow[WL];             // source rows, -1: none
  float4 xn[XL], wn[WL];

  __device__ __forceinline__ TileLoads(const int* row_index, int m0, int n0, int rows, int x_rows, int n, unsigned* status) {
#pragma unroll
    for (int i = 0; i < XL; ++i) {
      const int word = threadIdx.x + i * THREADS, r = m0 + word / WORDS;
      xrow[i] = -1;
      if (word < BM * WORDS && r < rows) {
        const int from = row_index ? row_index[r] : r;           // gathered for the LM head
        if (from < 0 || from >= x_rows) raise_fault(status, VOSTI_FAULT_ROW_RANGE);
        else xrow[i] = from;
      }
    }
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      const int word = threadIdx.x + i * THREADS, c = n0 + word / WORDS;
      wrow[i] = word < BN * WORDS && c < n ? c : -1;
    }
  }
  __device__ __forceinline__ void fetch(const TX* x, const TW* w, int k0, int k, bool wide) {
#pragma unroll
    for (int i = 0; i < WL; ++i) wn[i] = load4_of(w, wrow[i], k0 + ((threadIdx.x + i * THREADS) % WORDS) * 4, k, wide);
#pragma unroll
    for (int i = 0; i < XL; ++i) xn[i] = load4_of(x, xrow[i], k0 + ((threadIdx.x + i * THREADS) % WORDS) * 4, k, wide);
  }
  // store(row, first k of the word, its four values), for x and for w
  template <typename FX, typename FW>
  __device__ __forceinline__ void put(FX&& store_x, FW&& store_w) const {
#pragma unroll
    for (int i = 0; i < XL; ++i) {
      const int word = threadIdx.x + i * THREADS;
      if (BM * WORDS % THREADS == 0 || word < BM * WORDS) store_x(word / WORDS, (word % WORDS) * 4, xn[i]);
    }
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      const int word = threadIdx.x + i * THREADS;
      if (BN * WORDS % THREADS == 0 || word < BN * WORDS) store_w(word / WORDS, (word % WORDS) * 4, wn[i]);
    }
  }
};

// Few rows: the weights' way from memory bounds it, so a block takes few columns (many blocks, each with
// long words in flight) and both operands stay in shared memory as they lie, rows of BK + 4 floats (an odd
// number of 16-byte words: neighbouring rows in different banks). A thread computes TM x TN outputs, rows
// ty + i * (BM / TM), columns tx + j * (BN / TN).
template <typename TX, typename TW, typename TY, int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_few_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TY* __restrict__ y,
                     const int* __restrict__ row_index, int rows, int x_rows, int n, int k, int wide, unsigned* status) {
  constexpr int GX = BN / TN, GY = BM / TM, THREADS = GX * GY, PITCH = BK + 4;
  static_assert(BK % 8 == 0 && BM % TM == 0 && BN % TN == 0, "tile");
  __shared__ __align__(16) float xs[2][BM][PITCH];
  __shared__ __align__(16) float ws[2][BN][PITCH];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = threadIdx.x % GX, ty = threadIdx.x / GX;
  TileLoads<TX, TW, BM, BN, BK, THREADS> loads(row_index, m0, n0, rows, x_rows, n, status);
  auto put = [&](int buf) {
    loads.put([&](int r, int c, float4 v) { *reinterpret_cast<float4*>(&xs[buf][r][c]) = v; },
              [&](int r, int c, float4 v) { *reinterpret_cast<float4*>(&ws[buf][r][c]) = v; });
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  loads.fetch(x, w, 0, k, wide);
  put(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < k; k0 += BK, buf ^= 1) {
    const bool more = k0 + BK < k;
    if (more) loads.fetch(x, w, k0 + BK, k, wide);
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(&xs[buf][ty + i * GY][kk]);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(&ws[buf][tx + j * GX][kk]);
#pragma unroll
        for (int i = 0; i < TM; ++i)
          acc[i][j] = fmaf(a[i].w, b.w, fmaf(a[i].z, b.z, fmaf(a[i].y, b.y, fmaf(a[i].x, b.x, acc[i][j]))));
      }
    }
    if (more) put(buf ^ 1);             // (its last readers passed the barrier below)
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = m0 + ty + i * GY;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int c = n0 + tx + j * GX;
      if (c < n) y[(int64_t)r * n + c] = from_f32<TY>(acc[i][j]);
    }
  }
}

// Two rows' chains in one instruction.
typedef unsigned long long packed2;
__device__ __forceinline__ packed2 fma2(packed2 a, packed2 b, packed2 c) {
  packed2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ packed2 twice(float v) {
  packed2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}

// Many rows: the multiply-add pipe bounds it. Both operands are turned to [k][row] on their way into shared
// memory, so that a thread reads four neighbouring rows as one word and its 8 x TN outputs cost two words of
// x and TN / 4 of w a k; the packed multiply-add takes two neighbouring rows of x as they lie in that word.
// WIDE: every row of x and w starts on a whole word.
template <typename TX, typename TW, typename TY, int BM, int BN, int BK, int TN, int BLOCKS, bool WIDE>
__global__ void __launch_bounds__((BM / 8) * (BN / TN), BLOCKS)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TY* __restrict__ y,
                 const int* __restrict__ row_index, int rows, int x_rows, int n, int k, int, unsigned* status) {
  constexpr int GX = BN / TN, GY = BM / 8, THREADS = GX * GY;
  static_assert(BK % 4 == 0 && GX % 8 == 0 && GY % 4 == 0 && TN % 4 == 0, "tile");
  __shared__ __align__(16) float xs[2][BK][BM + 4];
  __shared__ __align__(16) float ws[2][BK][BN + 4];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = (warp % (GX / 8)) * 8 + lane % 8, ty = (warp / (GX / 8)) * 4 + lane / 8;
  TileLoads<TX, TW, BM, BN, BK, THREADS> loads(row_index, m0, n0, rows, x_rows, n, status);
  auto put = [&](int buf) {
    loads.put([&](int r, int c, float4 v) { xs[buf][c][r] = v.x; xs[buf][c + 1][r] = v.y; xs[buf][c + 2][r] = v.z; xs[buf][c + 3][r] = v.w; },
              [&](int r, int c, float4 v) { ws[buf][c][r] = v.x; ws[buf][c + 1][r] = v.y; ws[buf][c + 2][r] = v.z; ws[buf][c + 3][r] = v.w; });
  };
  packed2 acc[4][TN];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
  loads.fetch(x, w, 0, k, WIDE);
  put(0);
  __syncthreads();
  for (int k0 = 0, buf = 0; k0 < k; k0 += BK, buf ^= 1) {
    const bool more = k0 + BK < k;
    if (more) loads.fetch(x, w, k0 + BK, k, WIDE);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(&xs[buf][kk][ty * 4]);
      const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(&xs[buf][kk][BM / 2 + ty * 4]);
      const packed2 a[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
      for (int q = 0; q < TN / 4; ++q) {
        const float4 b = *reinterpret_cast<const float4*>(&ws[buf][kk][q * (BN * 4 / TN) + tx * 4]);
        const float bs[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const packed2 both = twice(bs[j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][q * 4 + j] = fma2(a[i], both, acc[i][q * 4 + j]);
        }
      }
    }
    if (more) put(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = m0 + (i / 4) * (BM / 2) + ty * 4 + i % 4;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int c = n0 + (j / 4) * (BN * 4 / TN) + tx * 4 + j % 4;
      const packed2 pair = acc[i / 2][j];
      if (c < n) y[(int64_t)r * n + c] = from_f32<TY>(__uint_as_float((unsigned)(i & 1 ? pair >> 32 : pair)));
    }
  }
}

template <typename TX, typename TW, typename TY>
void launch(const void* x, const void* w, void* y, const int* row_index, int rows, int x_rows, int n,
            int k, unsigned* status, cudaStream_t stream) {
  // words of four elements: every row starts on a whole word
  const int wide = k % 4 == 0 && reinterpret_cast<uintptr_t>(x) % (4 * sizeof(TX)) == 0 &&
                   reinterpret_cast<uintptr_t>(w) % (4 * sizeof(TW)) == 0;
#define VOSTI_SIMT(KERNEL, BM, BN, THREADS)                                                                           \
  KERNEL<<<dim3((n + BN - 1) / BN, (rows + BM - 1) / BM), THREADS, 0, stream>>>((const TX*)x, (const TW*)w, (TY*)y, \
                                                                               row_index, rows, x_rows, n, k, wide, status)
#define VOSTI_FEW(BM, BN, BK, TM, TN) VOSTI_SIMT((gemm_simt_few_kernel<TX, TW, TY, BM, BN, BK, TM, TN>), BM, BN, (BM / TM) * (BN / TN))
#define VOSTI_MANY(BM, BN, BK, TN, BLOCKS, WIDE) \
  VOSTI_SIMT((gemm_simt_kernel<TX, TW, TY, BM, BN, BK, TN, BLOCKS, WIDE>), BM, BN, (BM / 8) * (BN / TN))
  // Measured at float32, (n, k) = (4,096, 4,096) | (24,576, 4,096), us, against the 64 x 64 tile of 4 x 4 a thread that
  // this replaces: 1 row 27 | 156 (226 | 556), 8 rows 39 | 185 (229 | 568), 32 rows 77 | 268 (238 | 608), 100 rows
  // 187 | 695 (276 | 1,182), 384 rows 407 | 1,690 (621 | 3,123), 1,024 rows 868 | 4,242 (1,375 | 8,061; 49 TFLOP/s,
  // 0.65 of the multiply-add pipe). Where the lines lie: blocks of 8 columns cost 1.5 times as much from 5 rows on;
  // at 384 x 4,096 (192 tiles of 128 x 64) tiles of 64 x 32 take 407 and those of 128 x 64 490, at 384 x 6,144
  // (288 tiles) 555 and 484; at 100 x 4,096 (256 tiles of 64 x 32) 32 x 32 takes 187 and 64 x 32 245, at
  // 200 x 4,096 (512 tiles) 312 and 291. Rows that start inside a word (odd K) are loaded element by element, which a
  // larger tile does less often: the tile this replaces, 32 x 32 and 64 x 64 of 8 x 4 a thread, bfloat16: 384 x 4,096 x
  // 4,097 538, 678 and 430, 512 x 1,000 x 1,001 56, 69 and 53, 200 x 1,000 (128 tiles of 64 x 32) 56, 54 and 52;
  // float32: 1,000 x 4,096 x 4,097 1,170, 1,407 and 856.
  const int64_t columns = (n + 31) / 32;
  if (rows <= 4) VOSTI_FEW(4, 8, 256, 1, 1);
  else if (rows <= 8) VOSTI_FEW(8, 16, 128, 1, 1);
  else if (rows <= 16) VOSTI_FEW(16, 16, 64, 2, 1);
  else if (rows <= 32 || (rows <= 64 && columns < 3 * 148) || (rows + 63) / 64 * columns < (wide ? 3 : 1) * 148) VOSTI_FEW(32, 32, 32, 4, 2);
  else if (!wide) VOSTI_MANY(64, 64, 16, 4, 4, false);
  else if (rows <= 64 || (rows + 127) / 128 * ((columns + 1) / 2) < 288) VOSTI_MANY(64, 32, 16, 4, 10, true);
  else VOSTI_MANY(128, 64, 16, 8, 4, true);
#undef VOSTI_MANY
#undef VOSTI_FEW
#undef VOSTI_SIMT
}

}  // namespace

// x: [x_rows, k]; w: [n, k]; y: [rows, n]. With row_index (int32[rows]) row t of the
// product is taken from x[row_index[t]]; without it rows == x_rows.
VOSTI_API int vosti_gemm_simt(const void* x, const void* w, void* y, const int* row_index, int rows,
                              int x_rows, int n, int k, int x_is_f32, int w_is_f32, int y_is_f32,
                              unsigned* status, cudaStream_t stream) {
  VOSTI_REQUIRE(rows >= 0 && n > 0 && k > 0 && x_rows >= 0, "gemm: bad sizes rows=%d n=%d k=%d", rows, n, k);
  VOSTI_REQUIRE(row_index != nullptr || rows == x_rows, "gemm: rows != x_rows without a row index");
  if (rows == 0) return VOSTI_OK;
  VOSTI_REQUIRE((rows + 63) / 64 <= 65535, "gemm: too many rows (%d) for one launch", rows);
  const int code = (x_is_f32 ? 4 : 0) | (w_is_f32 ? 2 : 0) | (y_is_f32 ? 1 : 0);
  switch (code) {
    case 0: launch<bf16, bf16, bf16>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    case 1: launch<bf16, bf16, float>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    case 2: launch<bf16, float, bf16>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    case 3: launch<bf16, float, float>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    case 4: launch<float, bf16, bf16>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    case 5: launch<float, bf16, float>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    case 6: launch<float, float, bf16>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
    default: launch<float, float, float>(x, w, y, row_index, rows, x_rows, n, k, status, stream); break;
  }
  VOSTI_LAUNCH_CHECK();
}
