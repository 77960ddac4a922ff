// C[M,N] = A[M,K] . W[N,K]^T in true 32-bit.  The reference runs its 32-bit path through a library product
// with TF32 switched off (engine/engine.py:190-192); here the precision is a property of the code.
//
// A row's result does not depend, bit for bit, on which other rows share the launch: every form that a layout and K
// can take sums in one order, whatever M is.
//
// Rows of whole 32-byte pieces (K and both strides multiples of 8): tcgen05.  2^24 times a 32-bit value is the sum of three
// bfloat16 terms exactly (unscaled, the last terms of values below 2^-110 would lie below what bfloat16 holds), and the
// products of two terms are exact in 32 bits; the sums are scaled back at the end.  Values from 2^104 on and sums from 2^80 on
// go beyond 32 bits that way, see plain_sum.  Of the nine products of two values'
// terms the three smallest (2^-24 of the value and less) are left out; weights that came from 16 bits have one term,
// and then nothing is.  The tensor cores cut a sum at its last place instead of rounding it, so no more than 32 of K go
// into one accumulator: chunks of 32 are added in 32-bit registers, rounded, to spans of 256, and the spans to the result.
// Relative error against 64 bits (normal values, K = 1,024; this and FFMA in chains of 64): 0.9e-7 and 1.6e-7.
//   up to 64 rows   bound by the weight stream.  TMA brings 32-bit values, 16 warps write their terms for the MMA,
//                   the weights on its 128-row side; blocks take tile after tile, or a cluster shares K of one and
//                   every block sends its spans' sums to the one that adds them up.  us one behind the other in a graph, FFMA
//                   before, weights of one term (of three): 4 x 1024 x 3072 (M x N x K) 17.5 -> 11.3 (16.1), 16 x
//                   151936 x 1024 248 -> 112 (163; 5.6 TB/s), 13 x 6144 x 2560 78 -> 23 (36), 64 x 6144 x 2560 163 -> 37 (53).
//                   One row of a narrow product is the exception: 1 x 4096 x 1024 6.1 -> 9.7, the chain from copy to
//                   conversion, MMA and sum being longer than FFMA's.  Loads into registers or
//                   cp.async instead of TMA ran at half this rate (long chains in every converting warp).  Up to 8 rows by
//                   mma.sync from registers, whose results were the same bits, took 6.5 us there, but in a step, where small
//                   kernels stand between the products, 1.8 us more a product than this form.
//   more rows       a kernel of its own writes both operands' terms as the tiles that the MMA reads, so that a value is
//                   converted once and not by every block that needs it (which took half as long again); the product
//                   streams these tiles.  128 x 128 outputs a tile read 64 KB of operands for 64 of K (96 KB with three
//                   terms of the weights), two or three such stages in flight: ncu shows tensor pipes 34 % active and L2 at
//                   10.7 TB/s, 31 % of its sectors' peak, so neither is full.  1129 x 6144 x 1024 360 -> 87 us, 1129 x 1024 x 3072 219 -> 56,
//                   4096^3 3,165 -> 515 (267 TFLOP/s).  The three terms of x side by side in one MMA of 192 columns
//                   read less shared memory but more L2 (128 x 64 tiles): 820 us.
// Other rows, and K above 131,072: FFMA, chains of 64 (kRun) whose sums are added in ascending order.
//   few rows (M <= 16)  a lane takes a few columns and one run of K; one thread an output adds the runs' sums in order.
//   more rows           8 x 8 outputs a thread from tiles in shared memory.
#include "tc_common.cuh"

namespace ek {

constexpr int kRun = 64;              // products summed in one chain

// 8 values of a row from column k on (zeros from K on).
__device__ __forceinline__ void load8(float (&v)[8], const float* row, int k, int K) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = k + j < K ? row[k + j] : 0.f;
}

// ------------------------------------------------------------------------------- few rows
// Columns a lane: every x value that it fetches serves them all.
__host__ __device__ constexpr int few_cols(int mr) { return mr == 1 ? 1 : mr <= 4 ? 2 : 4; }
__host__ __device__ constexpr int few_warps(int mr) { return mr <= 8 ? 8 : 4; }      // (the runs' sums fit 48 KB)

// MR rows (M <= MR).  Lane = 8 groups of columns x 4 runs; a warp takes 4 runs at a time.
template <int MR>
__global__ void __launch_bounds__(few_warps(MR) * 32)
sgemm_few_rows_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                      int M, int N, int K, int lda, int ldw, int ldc) {
  constexpr int CPL = few_cols(MR), COLS = 8 * CPL;
  __shared__ float sums[few_warps(MR) * 4][COLS * MR + 1];
  __shared__ float totals[COLS * MR];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int runs_a_pass = (blockDim.x >> 5) * 4;
  const int n0 = blockIdx.x * COLS;
  const int group = lane & 7, my_run = warp * 4 + (lane >> 3);
  const float* w_row[CPL];                                // columns group, group + 8, ...
#pragma unroll
  for (int c = 0; c < CPL; ++c) w_row[c] = W + (size_t)min(n0 + c * 8 + group, N - 1) * ldw;
  const int total_runs = (K + kRun - 1) / kRun;
  for (int r0 = 0; r0 < total_runs; r0 += runs_a_pass) {
    const int k0 = (r0 + my_run) * kRun;
    if (k0 < K) {
      float acc[CPL][MR];
#pragma unroll
      for (int c = 0; c < CPL; ++c)
#pragma unroll
        for (int m = 0; m < MR; ++m) acc[c][m] = 0.f;
      constexpr int AHEAD = CPL == 4 ? 2 : kRun / 8 / CPL;  // 8-value pieces of a column asked for at once
#pragma unroll
      for (int i0 = 0; i0 < kRun / 8; i0 += AHEAD) {
        float w[CPL][AHEAD][8];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
#pragma unroll
          for (int c = 0; c < CPL; ++c) load8(w[c][i], w_row[c], k0 + 8 * (i0 + i), K);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
#pragma unroll
          for (int m = 0; m < MR; ++m) {
            float x[8];
            load8(x, A + (size_t)min(m, M - 1) * lda, k0 + 8 * (i0 + i), K);
#pragma unroll
            for (int c = 0; c < CPL; ++c)
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[c][m] = fmaf(x[j], w[c][i][j], acc[c][m]);
          }
      }
#pragma unroll
      for (int c = 0; c < CPL; ++c)
#pragma unroll
        for (int m = 0; m < MR; ++m) sums[my_run][(c * 8 + group) * MR + m] = acc[c][m];
    }
    __syncthreads();
    const int here = min(runs_a_pass, total_runs - r0);
    for (int o = tid; o < COLS * MR; o += blockDim.x) {    // (an output is one thread's in every pass)
      float t = r0 > 0 ? totals[o] : 0.f;
      for (int r = 0; r < here; ++r) t += sums[r][o];
      totals[o] = t;
      const int gm = o % MR, gn = n0 + o / MR;
      if (r0 + runs_a_pass >= total_runs && gm < M && gn < N) C[(size_t)gm * ldc + gn] = t;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------ more rows
// (A stage is written by plain stores three steps ahead of its use: rows here start anywhere, so there is nothing to copy
// 16 bytes at a time, and one barrier a step serves both the stage that is read and the one that is written.)
constexpr int kStepK = 16, kStepLd = kStepK + 4, kStages = 4;
__host__ __device__ constexpr int tile_smem(int bm, int bn) { return kStages * (bm + bn) * kStepLd * 4; }

// 8 x 8 outputs a thread: rows ty + i TY, columns tx + j TX.
template <int BM, int BN>
__global__ void __launch_bounds__(BM / 8 * (BN / 8))
sgemm_tile_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                  int M, int N, int K, int lda, int ldw, int ldc) {
  constexpr int TY = BM / 8, TX = BN / 8, THREADS = TX * TY;
  extern __shared__ __align__(16) float ring[];            // [stage][BM rows of A, BN rows of W][kStepLd]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // a warp's lanes: LY rows x LX columns (strided rows 20 floats apart: 16-byte reads without bank conflicts)
  constexpr int LY = TY < 4 ? TY : 4, LX = 32 / LY, WX = TX / LX;
  const int tx = warp % WX * LX + lane % LX, ty = warp / WX * LY + lane / LX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  auto copy = [&](int step) {
    float* to = ring + (size_t)(step % kStages) * (BM + BN) * kStepLd;
    const int k0 = step * kStepK;
#pragma unroll
    for (int p = 0; p < ((BM + BN) * (kStepK / 4) + THREADS - 1) / THREADS; ++p) {
      const int piece = tid + p * THREADS, row = piece / (kStepK / 4), k = k0 + piece % (kStepK / 4) * 4;
      if ((BM + BN) * (kStepK / 4) % THREADS && row >= BM + BN) break;
      const bool is_a = row < BM;
      const int r = is_a ? m0 + row : n0 + row - BM;
      const bool ok = r < (is_a ? M : N);
      const float* src = is_a ? A + (size_t)(ok ? r : 0) * lda : W + (size_t)(ok ? r : 0) * ldw;
      float* dst = to + row * kStepLd + piece % (kStepK / 4) * 4;
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[j] = ok && k + j < K ? src[k + j] : 0.f;
    }
  };

  float acc[8][8], total[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = total[i][j] = 0.f;

  const int steps = (K + kStepK - 1) / kStepK;
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) copy(s);
  }
  for (int s = 0; s < steps; ++s) {
    __syncthreads();                           // the step's operands are there, and the stage refilled below is free
    if (s + kStages - 1 < steps) copy(s + kStages - 1);
    const float* a_s = ring + (size_t)(s % kStages) * (BM + BN) * kStepLd + ty * kStepLd;
    const float* w_s = ring + (size_t)(s % kStages) * (BM + BN) * kStepLd + (BM + tx) * kStepLd;
#pragma unroll
    for (int k = 0; k < kStepK; k += 4) {
      float a[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(a[i]) = *reinterpret_cast<const float4*>(a_s + i * TY * kStepLd + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 w = *reinterpret_cast<const float4*>(w_s + j * TX * kStepLd + k);
        const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(a[i][kk], wv[kk], acc[i][j]);
      }
    }
    if ((s + 1) % (kRun / kStepK) == 0 || s + 1 == steps) {  // the end of a run of 64
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          total[i][j] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gm = m0 + ty + i * TY;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int gn = n0 + tx + j * TX;
      if (gn < N) C[(size_t)gm * ldc + gn] = total[i][j];
    }
  }
}

template <int BM, int BN>
static int launch_tile(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc,
                       cudaStream_t stream) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return EK_ERR_ARG;
  auto kernel = sgemm_tile_kernel<BM, BN>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem(BM, BN));
  if (e != cudaSuccess) return (int)e;
  kernel<<<grid, BM / 8 * (BN / 8), tile_smem(BM, BN), stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
  return (int)cudaGetLastError();
}

static int launch_ffma(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  // 9 to 16 rows of many columns: x is read often enough for the few-row form to be bound by L1, and there are columns
  // enough for tiles of 16 x 128 (us, few-row form / tiles: 16 x 40000 x 1025 224 / 165, 12 x 151936 x 1025 713 / 490; but
  // 16 x 24576 x 1025 137 / 160, 16 x 6144 x 1025 47 / 106, 8 x 151936 x 1025 366 / 489)
  if (M <= 16 && !(M > 8 && N > 28672)) {
    const int mr = M == 1 ? 1 : M <= 4 ? 4 : M <= 8 ? 8 : 16;
    const int threads = 32 * min(few_warps(mr), (K + 4 * kRun - 1) / (4 * kRun));
    const dim3 grid((N + 8 * few_cols(mr) - 1) / (8 * few_cols(mr)));
    if (mr == 1) sgemm_few_rows_kernel<1><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    else if (mr == 4) sgemm_few_rows_kernel<4><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    else if (mr == 8) sgemm_few_rows_kernel<8><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    else sgemm_few_rows_kernel<16><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    return (int)cudaGetLastError();
  }
  if (M <= 16) return launch_tile<16, 128>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  return launch_tile<64, 64>(C, A, W, M, N, K, lda, ldw, ldc, stream);
}

// ------------------------------------------------------------------------- on the tensor cores
constexpr int kSpan = 256;            // of K: a span's sum is that of its chunks of 32, a result that of its spans
constexpr int kStepSpan = kSpan / 64;
constexpr int kTermTile = 128 * 128;  // bytes of one term of 128 rows, 64 of K

// 8 values, 2^24 times as large, as sums of three bfloat16 terms each, exactly: x = hi + mid + lo, every term the nearest to
// what the ones before it leave; the last bit of the smallest 32-bit number is 2^-125 then, a normal one.  (Of an infinity, a
// NaN, or a value that rounds to an infinity in 16 bits the third is a NaN, see plain_sum.)
constexpr float kScaleBack = 0x1p-48f;
__device__ __forceinline__ void scale_up(float (&v)[8]) {
  const uint64_t by = 0x4b8000004b800000ull;                     // 2^24, twice
#pragma unroll
  for (int i = 0; i < 8; i += 2)
    asm("{.reg .b64 p; mov.b64 p, {%0, %1}; mul.rn.f32x2 p, p, %2; mov.b64 {%0, %1}, p;}" : "+f"(v[i]), "+f"(v[i + 1]) : "l"(by));
}
__device__ __forceinline__ uint32_t two_bf16(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ uint4 first_terms(const float (&v)[8]) {
  return make_uint4(two_bf16(v[0], v[1]), two_bf16(v[2], v[3]), two_bf16(v[4], v[5]), two_bf16(v[6], v[7]));
}
__device__ __forceinline__ void other_terms(const float (&v)[8], const uint4& hi, uint4& mid, uint4& lo) {
  const uint32_t h[4] = {hi.x, hi.y, hi.z, hi.w};
  uint32_t m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = v[2 * i] - __uint_as_float(h[i] << 16), b = v[2 * i + 1] - __uint_as_float(h[i] & 0xffff0000u);
    m[i] = two_bf16(a, b);
    l[i] = two_bf16(a - __uint_as_float(m[i] << 16), b - __uint_as_float(m[i] & 0xffff0000u));
  }
  mid = make_uint4(m[0], m[1], m[2], m[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ void load_row8(float (&v)[8], const float* from, bool there) {
  if (there) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(from));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
  }
}
__device__ __forceinline__ void st_shared_16(uint32_t at, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// One output by FFMA, in the order of chunks and spans.  It takes the place of a result of the terms that is not finite,
// which tells two kinds of outputs: those that an infinity or a NaN belongs to, and those of a row with a value, or of
// sums, that scaled up are one (2^104 and 2^80).  The terms of all these values give a NaN or an infinity, here in the wrong place or not: the
// third term of x is a NaN then, and is multiplied with every row of the weights; weights of one term only are an infinity
// or a NaN themselves, times three terms of x of which one is zero or all are not.  So nothing has to be looked for while
// terms are written, and only such rows' (and columns') outputs cost more.  (A flag for the block, and every output of its
// tiles worked out again to see whether its rows were the ones, took 1,100 x 4096 x 2048 with one infinity from 0.14 to
// 36 ms.)  A sum that is a NaN stays one.  (Inlined: as a function of its own it costs the kernels registers.)
__device__ __forceinline__ float plain_sum(const float* a, const float* w, int K) {
  float total = 0.f, span = 0.f;
#pragma unroll 1
  for (int c = 0; c < K; c += 32) {
    float x[4][8], y[4][8], chunk = 0.f;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      load_row8(x[p], a + c + 8 * p, c + 8 * p < K);
      load_row8(y[p], w + c + 8 * p, c + 8 * p < K);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int j = 0; j < 8; ++j) chunk = fmaf(x[p][j], y[p][j], chunk);
    span += chunk;
    if (span != span) return span;
    if ((c + 32) % kSpan == 0 || c + 32 >= K) {
      total += span;
      span = 0.f;
    }
  }
  return total;
}
__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) < INFINITY; }
// The outputs from `c` on, `count` rows of one column, that are not finite.
__device__ __forceinline__ void plain_where_not_finite(float* c, const float* a, const float* w, int count, int K, int lda, int ldc) {
#pragma unroll 1
  for (int m = 0; m < count; ++m, a += lda, c += ldc)
    if (!is_finite(*c)) *c = plain_sum(a, w, K);
}

// The MMAs of one chunk of 32 (c: the stage's first or second) into the NT columns from `acc` on; tile(i) is where
// term i (0-2 the weights', 3-5 x's) of the stage begins.  `more`: the weights have second or third terms.  The
// smallest products come first: the tensor cores cut a sum, rather than round it, at the last place it holds (a
// chain of 64 by 4.5e-8 of it on average, of 1,024 by 8e-7).
template <int NT, typename Tile>
__device__ __forceinline__ void chunk_mmas(uint32_t acc, Tile tile, int c, bool more) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  auto product = [&](int w, int x, uint32_t add) {
    const uint64_t wd = smem_desc_k_sw128(tile(w)) + 4 * c, xd = smem_desc_k_sw128(tile(3 + x)) + 4 * c;
    tc_mma(acc, wd, xd, idesc, add);
    tc_mma(acc, wd + 2, xd + 2, idesc, 1u);
  };
  if (more) {
    product(2, 0, 0);
    product(1, 1, 1);
    product(0, 2, 1);
    product(1, 0, 1);
  } else {
    product(0, 2, 0);
  }
  product(0, 1, 1);
  product(0, 0, 1);
}

// ------------------------------------------------------------- few rows: operands converted on their way in
constexpr int kConvWarps = 16, kAddWarps = 4, kFewThreads = (kConvWarps + kAddWarps + 3) * 32;
// Shared memory of a block: two stages of first terms of the weights and all of x's, the weights' other terms (of one
// stage where K is split: those blocks are short and want their values early), `depth` stages of values as they are,
// sums that other blocks send.
constexpr int kTermStages = 2;
__host__ __device__ constexpr int few_terms(int nt) { return kTermTile + 3 * nt * 128; }
__host__ __device__ constexpr int few_low(bool split) { return (split ? 1 : kTermStages) * 2 * kTermTile; }
__host__ __device__ constexpr int few_raw(int nt) { return (128 + nt) * 256; }
constexpr int kFewDepth = 4;
__host__ __device__ constexpr int few_fixed(int nt, bool split) {           // (barriers; a 1024-byte border)
  return kTermStages * few_terms(nt) + few_low(split) + 512 + 1024;
}
constexpr int kMaxSmem = 227 * 1024;

__device__ __forceinline__ void read_16(float* v, uint32_t at) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
}

// C tiles of 128 columns (weight rows, the MMA's M) x NT rows (tokens, its N).  SPLIT: the blocks of a cluster
// share K of one tile, whole spans each; otherwise a block takes tile after tile.
template <int NT, bool SPLIT>
__global__ void __launch_bounds__(kFewThreads, 1)
sgemm_tc_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                 int M, int N, int K, int lda, int ldw, int ldc, int spans_a_block,
                 int depth, int* status) {
  constexpr int CW = kConvWarps, AW = kAddWarps;
  constexpr uint32_t kStage = few_terms(NT), kRaw = few_raw(NT), kXTile = NT * 128;
  extern __shared__ unsigned char raw[];
  unsigned char* ring = raw + ((1024 - (smem_u32(raw) & 1023)) & 1023);
  const uint32_t terms0 = smem_u32(ring), low0 = terms0 + kTermStages * kStage, raw0 = low0 + few_low(SPLIT);
  unsigned char* tail = ring + kTermStages * kStage + few_low(SPLIT) + depth * kRaw;
  uint64_t* bars = (uint64_t*)tail;                     // full[2], summed[2], taken[2], done, received, here[4], read[4]
  uint32_t* tmem_slot = (uint32_t*)(bars + 16);
  unsigned char* more_terms = (unsigned char*)(tmem_slot + 4);     // [stage][CW]: the weights have second or third terms
  float* received = (float*)(tail + 512);               // [span][token of this block][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.z * NT, tiles_n = (N + 127) / 128;
  const int k_begin = SPLIT ? blockIdx.y * spans_a_block * kSpan : 0;
  const int k_end = SPLIT ? min(K, k_begin + spans_a_block * kSpan) : K;
  const int stages = k_end > k_begin ? (k_end - k_begin + 63) / 64 : 0;
  const int tiles = SPLIT ? 1 : (tiles_n - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int total = tiles * stages;
  const uint32_t full0 = smem_u32(bars), summed0 = full0 + 16, taken0 = full0 + 32, done = full0 + 48,
                 received0 = full0 + 56, here0 = full0 + 64, read0 = full0 + 96;
  // split: block r of the cluster adds up the tokens r, r + ranks, ...
  const int rank = SPLIT ? blockIdx.y : 0, ranks = SPLIT ? gridDim.y : 1, rows = min(NT, M - m0);
  const int slots = (rows + ranks - 1) / ranks, mine = rows > rank ? (rows - rank + ranks - 1) / ranks : 0;
  const int all_spans = (K + kSpan - 1) / kSpan;

  // The copying thread has its own barriers ready and the first weights on their way before anything else, and
  // before the kernel ahead has ended: weights do not depend on it.
  const uint64_t once = l2_policy_evict_first();
  auto raw_at = [&](int slot) { return raw0 + (uint32_t)slot * kRaw; };
  auto copy_w = [&](int slot, int tile, int s) {
    mbar_expect_tx(here0 + 8 * slot, kRaw);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      tma_load_2d_hint(raw_at(slot) + h * (128 * 128), &map_w, k_begin + s * 64 + h * 32, tile * 128, here0 + 8 * slot, once);
  };
  auto copy_x = [&](int slot, int s) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      tma_load_2d(raw_at(slot) + 128 * 256 + h * (NT * 128), &map_x, k_begin + s * 64 + h * 32, m0, here0 + 8 * slot);
  };
  pdl_launch_dependents();
  if (tid == (AW + CW) * 32) {
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_x);
    for (int i = 0; i < depth; ++i) {
      mbar_init(here0 + 8 * i, 1);
      mbar_init(read0 + 8 * i, CW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int q = 0; q < min(depth, total); ++q) copy_w(q, blockIdx.x + q / stages * gridDim.x, q % stages);
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(full0 + 8 * i, CW);
      mbar_init(summed0 + 8 * i, 2);
      mbar_init(taken0 + 8 * i, AW);
    }
    mbar_init(done, 2);
    mbar_init(received0, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (SPLIT && mine > 0) mbar_expect_tx(received0, (uint32_t)(all_spans * mine * 512));
  }
  // (that barrier exists in every block before a store from another one reaches it: arrive here, wait before the
  // first such store)
  __syncwarp();
  if (SPLIT) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  if (warp == AW + CW) tmem_alloc(smem_u32(tmem_slot), 8 * NT);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lanes = tmem + ((uint32_t)(warp * 32) << 16);
  bool ok = true;
  if (warp < AW) pdl_wait();                               // before anything is written

  if (warp < AW) {
    // ------------------------------------------------------------------ chunk sums out of TMEM, added in 32 bits
    float span[NT];
    int s = 0, tile = blockIdx.x;
    if (SPLIT) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll 1
    for (int q = 0; q < total; ++q) {
      if (!(ok = mbar_wait(summed0 + 8 * (q & 1), (q >> 1) & 1, status, 33))) break;
      tc_fence_after();
      const bool fresh = s % kStepSpan == 0;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int t = 0; t < NT; t += 16) {
          float v[16];
          tmem_ld16(lanes + (uint32_t)((2 * (q & 1) + c) * NT + t), v);
#pragma unroll
          for (int j = 0; j < 16; ++j) span[t + j] = c == 0 && fresh ? v[j] : span[t + j] + v[j];
        }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(taken0 + 8 * (q & 1));
      const bool last = ++s == stages;
      if (s % kStepSpan != 0 && !last) continue;
      const int span_of = (s - 1) / kStepSpan;
      if constexpr (SPLIT) {
        // every token's sum to the block that adds it up
        const int at = k_begin / kSpan + span_of;
        int to = 0, slot = 0;
#pragma unroll
        for (int t = 0; t < NT; ++t)
          if (t < rows) {
            st_async_f32(&received[((size_t)at * slots + slot) * 128 + tid], (unsigned)to, span[t], received0);
            if (++to == ranks) {
              to = 0;
              ++slot;
            }
          }
      } else {
        // the total of the spans so far waits in tensor memory
#pragma unroll
        for (int t = 0; t < NT; t += 16) {
          if (span_of > 0) {
            float v[16];
            tmem_ld16(lanes + (uint32_t)(4 * NT + t), v);
#pragma unroll
            for (int j = 0; j < 16; ++j) span[t + j] = v[j] + span[t + j];
          }
          if (!last) {
            uint32_t v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(span[t + j]);
            tmem_st16(lanes + (uint32_t)(4 * NT + t), v);
          }
        }
        tmem_st_wait();
        if (last) {
          s = 0;
          const int n = tile * 128 + tid;
          bool finite = true;
#pragma unroll
          for (int t = 0; t < NT; ++t)
            if (n < N && t < rows) {
              C[(size_t)(m0 + t) * ldc + n] = span[t] * kScaleBack;
              finite = finite && is_finite(span[t]);
            }
          if (!finite) plain_where_not_finite(C + (size_t)m0 * ldc + n, A + (size_t)m0 * lda, W + (size_t)n * ldw, rows, K, lda, ldc);
          tile += gridDim.x;
        }
      }
    }
    if (SPLIT && ok && mine > 0) {
      ok = mbar_wait(received0, 0, status, 39);
      const int n = blockIdx.x * 128 + tid;
      if (ok && n < N)
        for (int i = 0; i < mine; ++i) {
          float sum = 0.f;
#pragma unroll 4
          for (int j = 0; j < all_spans; ++j) {
            const float v = received[((size_t)j * slots + i) * 128 + tid];
            sum = j > 0 ? sum + v : v;
          }
          const size_t m = m0 + rank + i * ranks;
          C[m * ldc + n] = is_finite(sum) ? sum * kScaleBack : plain_sum(A + m * lda, W + (size_t)n * ldw, K);
        }
    }
  } else if (warp < AW + CW) {
    // ------------------------------------------------------------------- three terms of each value to shared memory
    // A pass is 8 rows x 32 of K, 8 values a lane; a warp takes two of the weights and where there are some left one
    // of x.  Neighbouring fours of lanes take rows r and r ^ 5: 16-byte accesses to the swizzled rows of either side
    // then touch every bank once.
    // Weights that came from 16 bits have a first term only: the others are written where they are not zero, or
    // where such were before.
    const int cw = warp - AW, i8 = lane >> 2, r8 = (i8 >> 1) ^ (i8 & 1 ? 5 : 0), k4 = lane & 3;
    const bool has_x = cw < NT / 4;
    const uint32_t even = (uint32_t)(((2 * k4) ^ r8) << 4), odd = even ^ 16u;
    uint32_t to_w[2];                                     // where a pass's first terms go, from the stage's start on
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int n = cw + p * CW;
      to_w[p] = (8 * (n >> 1) + r8) * 128 + (((4 * (n & 1) + k4) ^ r8) << 4);
      for (int i = 0; i < (SPLIT ? 2 : 4); ++i) st_shared_16(low0 + i * kTermTile + to_w[p], make_uint4(0, 0, 0, 0));
    }
    const uint32_t to_x = kTermTile + (8 * (cw >> 1) + r8) * 128 + (((4 * (cw & 1) + k4) ^ r8) << 4);
    uint32_t stale = 0;                                   // a bit each place of other terms: it holds some that are not zero
    int slot = 0, phase = 0;
#pragma unroll 1
    for (int q = 0; q < total; ++q) {
      if (!(ok = mbar_wait(here0 + 8 * slot, phase, status, 37))) break;
      const uint32_t from = raw0 + (uint32_t)slot * kRaw, at = terms0 + (q & 1) * kStage;
      float w[2][8], x[8];
      uint32_t low = 0, low_x = 0;
      // pass n: half n & 1 of the stage's K, rows 8 (n >> 1) ..
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int n = cw + p * CW;
        const uint32_t in = from + (n & 1) * (128 * 128) + (8 * (n >> 1) + r8) * 128;
        read_16(w[p], in + even);
        read_16(w[p] + 4, in + odd);
#pragma unroll
        for (int j = 0; j < 8; ++j) low |= __float_as_uint(w[p][j]);
      }
      if (has_x) {
        const uint32_t in = from + 128 * 256 + (cw & 1) * (NT * 128) + (8 * (cw >> 1) + r8) * 128;
        read_16(x, in + even);
        read_16(x + 4, in + odd);
#pragma unroll
        for (int j = 0; j < 8; ++j) low_x |= __float_as_uint(x[j]);
      }
      uint4 hi[2], x_hi;
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        scale_up(w[p]);
        hi[p] = first_terms(w[p]);
      }
      if (has_x) {
        scale_up(x);
        x_hi = first_terms(x);
      }
      const uint32_t with_more = __ballot_sync(0xffffffffu, (low & 0xffffu) != 0);
      const bool more = with_more != 0;
      // The place may be filled again once every lane has what it asked for.  Nothing but the need for the values keeps an
      // arrival behind reads that are on their way (neither a fence nor a barrier of the warp does: a form whose arrival had no use
      // for them found the values of the next filling in half of its rows), so which lane arrives is read from all of them.
      const uint32_t seen = with_more | (has_x ? __ballot_sync(0xffffffffu, (low_x & 0xffffu) != 0) : 0u);
      if (lane == 31 - __clz(seen | 1u)) mbar_arrive(read0 + 8 * slot);
      if (q >= kTermStages && !(ok = mbar_wait(summed0 + 8 * (q & 1), ((q >> 1) & 1) ^ 1, status, 31))) break;
#pragma unroll
      for (int p = 0; p < 2; ++p) st_shared_16(at + to_w[p], hi[p]);
      const int place = SPLIT ? 0 : q & 1;
      if (more || (stale >> place & 1)) {
        // (one place for both stages: the MMAs of the stage before have to be done)
        if (SPLIT && q > 0 && !(ok = mbar_wait(summed0 + 8 * ((q - 1) & 1), ((q - 1) >> 1) & 1, status, 31))) break;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          uint4 mid, lo;
          other_terms(w[p], hi[p], mid, lo);
          st_shared_16(low0 + place * 2 * kTermTile + to_w[p], mid);
          st_shared_16(low0 + place * 2 * kTermTile + to_w[p] + kTermTile, lo);
        }
      }
      stale = (stale & ~(1u << place)) | ((more ? 1u : 0u) << place);
      if (has_x) {
        uint4 mid, lo;
        st_shared_16(at + to_x, x_hi);
        other_terms(x, x_hi, mid, lo);
        st_shared_16(at + to_x + kXTile, mid);
        st_shared_16(at + to_x + 2 * kXTile, lo);
      }
      if (lane == 0) more_terms[(q & 1) * CW + cw] = more;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full0 + 8 * (q & 1));
      if (++slot == depth) {
        slot = 0;
        phase ^= 1;
      }
    }
  } else if (warp == AW + CW) {
    // ------------------------------------------------------------------------------ the values, DEPTH stages ahead
    if (lane == 0) {
      pdl_wait();
      int asked = min(depth, total), s = 0, tile = blockIdx.x, slot = 0, phase = 1;
#pragma unroll 1
      for (int q = 0; q < total; ++q) {
        if (q >= depth) {
          if (!(ok = mbar_wait(read0 + 8 * slot, phase, status, 38))) break;
          copy_w(slot, tile, s);
        }
        copy_x(slot, s);
        asked = max(asked, q + 1);
        if (++s == stages) {
          s = 0;
          tile += gridDim.x;
        }
        if (++slot == depth) {
          slot = 0;
          phase ^= 1;
        }
      }
      if (!ok)                                            // copies in flight land before the block leaves
        for (int q = max(0, asked - depth); q < asked; ++q) mbar_wait(here0 + 8 * (q % depth), (q / depth) & 1, status, 36);
    }
  } else if (lane == 0) {
    // ------------------------------------------------------------------------------------------- the MMAs
    // (two threads, a chunk of every stage each: a thread's barriers and commits take longer than its MMAs)
    const int c = warp - AW - CW - 1;
#pragma unroll 1
    for (int q = 0; q < total; ++q) {
      if (!(ok = mbar_wait(full0 + 8 * (q & 1), (q >> 1) & 1, status, 32))) break;
      if (q >= 2 && !(ok = mbar_wait(taken0 + 8 * (q & 1), ((q >> 1) & 1) ^ 1, status, 34))) break;
      tc_fence_after();
      uint4 more;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(more.x), "=r"(more.y), "=r"(more.z), "=r"(more.w)
                   : "r"(smem_u32(more_terms + (q & 1) * CW)) : "memory");
      const uint32_t base = terms0 + (q & 1) * kStage, low = low0 + (SPLIT ? 0 : (q & 1) * 2 * kTermTile);
      chunk_mmas<NT>(tmem + (uint32_t)((2 * (q & 1) + c) * NT),
                     [&](int i) { return i == 0 ? base : i < 3 ? low + (i - 1) * kTermTile : base + kTermTile + (i - 3) * kXTile; },
                     c, (more.x | more.y | more.z | more.w) != 0);
      tc_commit(summed0 + 8 * (q & 1));                    // with the other one's: the sums are there, and the stage may be filled again
    }
    tc_commit(done);                                      // every MMA that was issued has ended
    mbar_wait(done, 0, status, 35);
  }
  if (SPLIT) {
    // no block leaves while a sum may still be on its way to it, or before all have one that they wait for
    __syncwarp();
    if (warp >= AW) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == AW + CW) tmem_dealloc(tmem, 8 * NT);
  if (SPLIT) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Rows of 32-bit values, boxes of 32 x box_rows, 128-byte swizzle, zeros outside.
static bool tensor_map_f32(const float* rows, int n, int k, int ld, int box_rows, CUtensorMap* out) {
  const EncodeTiledFn fn = encode_fn();
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)n}, strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {32, (cuuint32_t)box_rows}, step[2] = {1, 1};
  return fn != nullptr && fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(rows), dims, strides, box, step,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How many clusters of b blocks run at a time (a GPU part's SMs are no multiple of b), asked once a device; 0 where it cannot
// be asked, this time.
template <int NT>
static int clusters_at_once(int b) {
  static std::mutex mu;
  static int counts[kMaxDevices][9] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return 0;
  std::lock_guard<std::mutex> lock(mu);
  int& count = counts[device][b];
  if (count > 0) return count;
  auto kernel = sgemm_tc_few_kernel<NT, true>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, b, 1);
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = kMaxSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = b;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) != cudaSuccess) {
    count = 0;
    cudaGetLastError();
  }
  return count;
}

template <int NT>
static int launch_few(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int* status,
                      cudaStream_t stream) {
  const int tiles_n = (N + 127) / 128, tiles_m = (M + NT - 1) / NT, spans = (K + kSpan - 1) / kSpan, sms = max(1, sm_count());
  if (tiles_m > 65535) return EK_ERR_ARG;
  // K over the blocks of a cluster where the tiles alone leave SMs idle: the fewest rounds of blocks, a block's cost
  // taken as its spans and one and a half for its start and end
  int blocks = 1, each = spans, kept = 0;
  const long long tiles = (long long)tiles_n * tiles_m;
  long long best = (tiles + sms - 1) / sms * (2 * spans) + 3;
  for (int b = 2; b <= 8 && b <= spans; ++b) {
    const int e = (spans + b - 1) / b, at_once = clusters_at_once<NT>(b);
    const long long sums = (long long)spans * ((min(NT, M) + b - 1) / b) * 512;
    if (at_once <= 0 || (b - 1) * e >= spans || sums > kMaxSmem - few_fixed(NT, true) - 2 * few_raw(NT)) continue;
    const long long cost = (tiles + at_once - 1) / at_once * (2 * e + 3);
    if (cost < best) {
      best = cost;
      blocks = b;
      each = e;
      kept = (int)sums;
    }
  }
  const bool split = blocks > 1;
  const int fits = (kMaxSmem - few_fixed(NT, split) - kept) / few_raw(NT), depth = fits < kFewDepth ? fits : kFewDepth;
  const int smem = few_fixed(NT, split) + kept + depth * few_raw(NT);
  auto kernel = split ? sgemm_tc_few_kernel<NT, true> : sgemm_tc_few_kernel<NT, false>;
  CUtensorMap map_w, map_x;
  if (!tensor_map_f32(W, N, K, ldw, 128, &map_w) || !tensor_map_f32(A, M, K, lda, NT, &map_x)) return EK_ERR_ARG;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid(split ? tiles_n : min(tiles_n, max(1, sms / tiles_m)), blocks, tiles_m);
  e = split ? launch_pdl_cluster(kernel, grid, dim3(kFewThreads), smem, stream, blocks, map_w, map_x, C, A, W, M, N, K, lda, ldw, ldc,
                                 each, depth, status)
            : launch_pdl(kernel, grid, dim3(kFewThreads), smem, stream, map_w, map_x, C, A, W, M, N, K, lda, ldw, ldc, each, depth, status);
  return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

// ------------------------------------------------------------------ many rows: operands converted ahead
// Images: [row block of 128][64 of K][term] tiles of 16 KB as the MMA reads them (K-major, 128-byte swizzle), and
// one word a (row block of the weights, 64 of K): whether there are second or third terms.

__global__ void __launch_bounds__(256)
sgemm_terms_kernel(uint4* __restrict__ images, uint32_t* __restrict__ flags, const float* __restrict__ A, const float* __restrict__ W,
                   int M, int N, int K, int lda, int ldw, int w_blocks) {
  const int tid = threadIdx.x, piece = tid & 7, row = tid >> 3, kb = blockIdx.x, rb = blockIdx.y;
  const bool is_w = rb < w_blocks;
  pdl_launch_dependents();
  const int r0 = (is_w ? rb : rb - w_blocks) * 128, limit = is_w ? N : M, k = kb * 64 + 8 * piece;
  const float* from = is_w ? W : A;
  const size_t ld = is_w ? ldw : lda;
  float v[4][8];
  uint32_t low = 0;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    load_row8(v[p], from + (size_t)(r0 + row + 32 * p) * ld + k, r0 + row + 32 * p < limit && k < K);
#pragma unroll
    for (int j = 0; j < 8; ++j) low |= __float_as_uint(v[p][j]);
  }
  const int more = __syncthreads_or((low & 0xffffu) != 0);
  uint4* to = images + ((size_t)rb * gridDim.x + kb) * (3 * kTermTile / 16) + row * 8 + (piece ^ (row & 7));
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    scale_up(v[p]);
    const uint4 hi = first_terms(v[p]);
    to[p * 256] = hi;
    if (more || !is_w) {                         // (the terms of x are always multiplied, also where they are zero)
      uint4 mid, lo;
      other_terms(v[p], hi, mid, lo);
      to[p * 256 + kTermTile / 16] = mid;
      to[p * 256 + 2 * kTermTile / 16] = lo;
    }
  }
  if (is_w && tid == 0) flags[(size_t)rb * gridDim.x + kb] = more ? 1u : 0u;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

constexpr int kManyThreads = 352;     // 8 warps that add, one that copies, two that issue MMAs
constexpr int kManyRing = 13;         // tiles of 16 KB: 3 stages of weights in one term, 2 in three
constexpr int kManySlots = 4;         // stages that barriers are kept for
constexpr int kManySmem = kManyRing * kTermTile + 512 + 1024;

// C tiles of 128 columns x NT rows; a block takes tile after tile.  A stage takes the tiles of the ring that it needs:
// the weights' first term or all three, then the three terms of x.  (128 rows a tile: an adding thread keeps 128 sums, and of
// the 168 registers that 11 warps leave it spills 160 bytes, 232 read back a tile's end and span; 64 rows spill nothing but
// stream half as much again for an output.)
template <int NT>
__global__ void __launch_bounds__(kManyThreads, 1)
sgemm_tc_many_kernel(float* __restrict__ C, const unsigned char* __restrict__ images, const uint32_t* __restrict__ flags,
                  const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K, int lda, int ldw, int ldc,
                  int w_blocks, int* status) {
  constexpr int COLS = NT / 2;                          // tokens an adding thread takes
  extern __shared__ unsigned char raw[];
  unsigned char* ring = raw + ((1024 - (smem_u32(raw) & 1023)) & 1023);
  uint64_t* bars = (uint64_t*)(ring + kManyRing * kTermTile);   // full[4], freed[4], summed[2], taken[2], done
  uint32_t* tmem_slot = (uint32_t*)(bars + 14);
  volatile int* more_terms = (int*)(tmem_slot + 2);     // of the stage behind each barrier
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int stages = (K + 63) / 64, all_tiles = w_blocks * ((M + NT - 1) / NT);
  const int tiles = (all_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, total = tiles * stages;
  const uint32_t full0 = smem_u32(bars), freed0 = full0 + 32, summed0 = full0 + 64, taken0 = full0 + 80, done = full0 + 96;
  if (tid == 0) {
    for (int i = 0; i < kManySlots; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(freed0 + 8 * i, 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(summed0 + 8 * i, 2);
      mbar_init(taken0 + 8 * i, 8);
    }
    mbar_init(done, 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) tmem_alloc(smem_u32(tmem_slot), 4 * NT);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;
  if (warp <= 8) pdl_wait();                              // before images are read and anything is written

  if (warp < 8) {
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * COLS);
    float span[COLS], sum[COLS];
    int s = 0, tile = blockIdx.x;
#pragma unroll 1
    for (int q = 0; q < total; ++q) {
      if (!(ok = mbar_wait(summed0 + 8 * (q & 1), (q >> 1) & 1, status, 33))) break;
      tc_fence_after();
      const bool fresh = s % kStepSpan == 0;
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int t = 0; t < COLS; t += 16) {
          float v[16];
          tmem_ld16(lanes + (uint32_t)((2 * (q & 1) + c) * NT + t), v);
#pragma unroll
          for (int j = 0; j < 16; ++j) span[t + j] = c == 0 && fresh ? v[j] : span[t + j] + v[j];
        }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(taken0 + 8 * (q & 1));
      const bool last = s + 1 == stages;
      if (s % kStepSpan == kStepSpan - 1 || last) {
#pragma unroll
        for (int t = 0; t < COLS; ++t) sum[t] = s < kStepSpan ? span[t] : sum[t] + span[t];
      }
      if (!last) { ++s; continue; }
      s = 0;
      const int n = tile % w_blocks * 128 + (warp & 3) * 32 + lane, m0 = tile / w_blocks * NT + (warp >> 2) * COLS;
      bool finite = true;
#pragma unroll
      for (int t = 0; t < COLS; ++t)
        if (n < N && m0 + t < M) {
          C[(size_t)(m0 + t) * ldc + n] = sum[t] * kScaleBack;
          finite = finite && is_finite(sum[t]);
        }
      if (!finite)
        plain_where_not_finite(C + (size_t)m0 * ldc + n, A + (size_t)m0 * lda, W + (size_t)n * ldw, min(COLS, M - m0), K, lda, ldc);
      tile += gridDim.x;
    }
  } else if (warp == 8) {
    if (lane == 0) {
      int s = 0, tile = blockIdx.x, at = 0, room = kManyRing, oldest = 0, asked = 0;
      uint32_t sizes = 0;                               // tiles of the stages in flight, 8 bits each, the oldest lowest
      size_t wi = (size_t)(tile % w_blocks) * stages, xi = (size_t)(w_blocks + tile / w_blocks * NT / 128) * stages;
      uint32_t w_flag = total > 0 ? flags[wi] : 0;
#pragma unroll 1
      for (int q = 0; q < total; ++q) {
        const bool more = w_flag != 0;
        const int need = more ? 6 : 4, slot = q % kManySlots;
        while (ok && (room < need || q - oldest >= kManySlots)) {
          ok = mbar_wait(freed0 + 8 * (oldest % kManySlots), (oldest / kManySlots) & 1, status, 31);
          room += sizes & 255;
          sizes >>= 8;
          ++oldest;
        }
        if (!ok) break;
        const unsigned char *w_from = images + wi * (3 * kTermTile),
                            *x_from = images + xi * (3 * kTermTile) + (tile / w_blocks * NT & 127) * 128;
        more_terms[slot] = more;
        const uint32_t bar = full0 + 8 * slot;
        mbar_expect_tx(bar, (uint32_t)((need - 3) * kTermTile + 3 * NT * 128));
        for (int i = 0; i < need - 3; ++i) {
          bulk_load(smem_u32(ring) + at * kTermTile, w_from + i * kTermTile, kTermTile, bar);
          at = at + 1 == kManyRing ? 0 : at + 1;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          bulk_load(smem_u32(ring) + at * kTermTile, x_from + i * kTermTile, NT * 128, bar);
          at = at + 1 == kManyRing ? 0 : at + 1;
        }
        sizes |= (uint32_t)need << (8 * (q - oldest));
        room -= need;
        asked = q + 1;
        ++wi;
        ++xi;
        if (++s == stages) {
          s = 0;
          tile += gridDim.x;
          wi = (size_t)(tile % w_blocks) * stages;
          xi = (size_t)(w_blocks + tile / w_blocks * NT / 128) * stages;
        }
        if (q + 1 < total) w_flag = flags[wi];          // (its latency passes behind the next wait)
      }
      if (!ok)                                          // copies in flight land before the block leaves
        for (int q = oldest; q < asked; ++q) mbar_wait(full0 + 8 * (q % kManySlots), (q / kManySlots) & 1, status, 36);
    }
  } else if (lane == 0) {
    // (two threads, a chunk of every stage each: a thread's barriers and commits take longer than its MMAs)
    const int c = warp - 9;
    int at = 0;
#pragma unroll 1
    for (int q = 0; q < total; ++q) {
      const int slot = q % kManySlots;
      if (!(ok = mbar_wait(full0 + 8 * slot, (q / kManySlots) & 1, status, 32))) break;
      if (q >= 2 && !(ok = mbar_wait(taken0 + 8 * (q & 1), ((q >> 1) & 1) ^ 1, status, 34))) break;
      tc_fence_after();
      const bool more = more_terms[slot] != 0;
      const int w_tiles = more ? 3 : 1;
      chunk_mmas<NT>(tmem + (uint32_t)((2 * (q & 1) + c) * NT),
                     [&](int i) {
                       const int j = at + (i < 3 ? i : w_tiles + i - 3);
                       return smem_u32(ring) + (uint32_t)(j >= kManyRing ? j - kManyRing : j) * kTermTile;
                     }, c, more);
      tc_commit(freed0 + 8 * slot);
      tc_commit(summed0 + 8 * (q & 1));
      at += w_tiles + 3;
      if (at >= kManyRing) at -= kManyRing;
    }
    tc_commit(done);
    mbar_wait(done, 0, status, 35);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 9) {
    __syncwarp();
    tmem_dealloc(tmem, 4 * NT);
  }
}

// Bytes of images and flags for `rows` rows of x or of weights.
static size_t terms_bytes(int rows, int K) {
  return (size_t)((rows + 127) / 128) * ((K + 63) / 64) * (3 * kTermTile + 4);
}

template <int NT>
static int launch_many(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, unsigned char* scratch,
                       int* status, cudaStream_t stream) {
  const int w_blocks = (N + 127) / 128, x_blocks = (M + 127) / 128, stages = (K + 63) / 64;
  uint32_t* flags = (uint32_t*)(scratch + (size_t)(w_blocks + x_blocks) * stages * (3 * kTermTile));
  if (w_blocks + x_blocks > 65535) return EK_ERR_ARG;
  sgemm_terms_kernel<<<dim3(stages, w_blocks + x_blocks), 256, 0, stream>>>((uint4*)scratch, flags, A, W, M, N, K, lda, ldw, w_blocks);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  auto kernel = sgemm_tc_many_kernel<NT>;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kManySmem);
  if (e != cudaSuccess) return (int)e;
  const int tiles = w_blocks * ((M + NT - 1) / NT);
  return (int)launch_pdl(kernel, dim3(min(tiles, max(1, sm_count()))), dim3(kManyThreads), kManySmem, stream, C, (const unsigned char*)scratch,
                         (const uint32_t*)flags, A, W, M, N, K, lda, ldw, ldc, w_blocks, status);
}

constexpr int kFewRows = 64;          // up to here operands are converted on their way in
constexpr long long kImageBytes = 128ll << 20;    // of weights, and of rows of x, that are converted at a time
constexpr int kMostK = 1 << 17;       // of K: one block of 128 rows stays below that (longer rows: FFMA)
static_assert((kMostK / 64) * (3ll * kTermTile + 4) <= kImageBytes, "a block's images");

// Rows whose images are made at a time: equal parts, whole blocks.
static int image_rows(int rows, int K) {
  const long long block = (long long)((K + 63) / 64) * (3 * kTermTile + 4), blocks = (rows + 127) / 128;
  const long long most = kImageBytes / block > 1 ? kImageBytes / block : 1, parts = (blocks + most - 1) / most;
  return (int)((blocks + parts - 1) / parts * 128);
}

static int launch_tc(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc,
                           unsigned char* scratch, int* status, cudaStream_t stream) {
  if (M > kFewRows) {
    if (scratch == nullptr) return EK_ERR_ARG;
    const int rows_m = min(M, image_rows(M, K)), rows_n = min(N, image_rows(N, K));
    // 64 rows a tile cost three quarters of what 128 do
    const int sms = max(1, sm_count());
    auto rounds = [&](int nt) { return ((long long)((rows_n + 127) / 128) * ((rows_m + nt - 1) / nt) + sms - 1) / sms; };
    const bool wide = 4 * rounds(128) <= 3 * rounds(64);
    for (int n = 0; n < N; n += rows_n)
      for (int m = 0; m < M; m += rows_m) {
        float* c = C + (size_t)m * ldc + n;
        const float *a = A + (size_t)m * lda, *w = W + (size_t)n * ldw;
        const int mm = min(rows_m, M - m), nn = min(rows_n, N - n);
        const int rc = wide ? launch_many<128>(c, a, w, mm, nn, K, lda, ldw, ldc, scratch, status, stream)
                            : launch_many<64>(c, a, w, mm, nn, K, lda, ldw, ldc, scratch, status, stream);
        if (rc != 0) return rc;
      }
    return 0;
  }
  return M > 16 ? launch_few<32>(C, A, W, M, N, K, lda, ldw, ldc, status, stream)
                : launch_few<16>(C, A, W, M, N, K, lda, ldw, ldc, status, stream);
}

}  // namespace ek

// Bytes that a product of these sizes wants for its operands' terms (0: none), 256 MB at most.
EK_EXPORT int ek_gemm_f32_scratch(int M, int N, int K) {
  if (M <= ek::kFewRows || N <= 0 || K <= 0 || K % 8 != 0 || K > ek::kMostK) return 0;
  return (int)(ek::terms_bytes(ek::image_rows(M, K), K) + ek::terms_bytes(ek::image_rows(N, K), K));
}

EK_EXPORT int ek_gemm_nt_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda,
                             int ldw, int ldc, void* scratch, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldc < N) return EK_ERR_ARG;
  // (a rule on the layout and K, not on M: a row's result does not depend on the rows beside it)
  const bool vec = K % 8 == 0 && K <= ek::kMostK && lda % 8 == 0 && ldw % 8 == 0 && ((uintptr_t)A & 31) == 0 && ((uintptr_t)W & 31) == 0;
  return vec ? ek::launch_tc(C, A, W, M, N, K, lda, ldw, ldc, (unsigned char*)scratch, status, stream)
             : ek::launch_ffma(C, A, W, M, N, K, lda, ldw, ldc, stream);
}
