// C[M,N] = A[M,K] . W[N,K]^T in true 32-bit: FFMA on the CUDA cores, no tensor-core
// mode of reduced precision anywhere.  The reference runs its 32-bit path through a
// library product with TF32 switched off (engine/engine.py:190-192); this kernel makes
// the precision a property of the code instead of a global flag.
//
// One order of summation for every output, whatever M is and whichever form below runs: the K
// products of a run of 64 (kRun) are summed in ascending k from zero, and the runs' sums are added
// in ascending order.  A row's result therefore does not depend, bit for bit, on which other rows
// share the launch, and few rows can spread K over many lanes.
//
//   few rows (M <= 16)  bound by the weight stream.  A lane takes a few columns and one run of K: their
//                       weights straight from memory, 32 bytes a load, the rows' x from L1; it leaves the
//                       run's sums in shared memory, where one thread an output adds them in order.
//                       Measured (us, the 16 x 128 tiles over all of K before): 4 x 4096 x 1024 (M x N x K)
//                       111 -> 12.3, 4 x 1024 x 3072 311 -> 18.8, 1 x 151936 x 1024 347 -> 113 (5.5 TB/s).
//   more rows           bound by the FMA pipes and the shared-memory reads that feed them: 8 x 8 outputs a
//                       thread read 16 values of 4 steps of K by 16-byte loads for 256 FMAs, which takes
//                       shared memory as long as the FMAs take (a warp's 16-byte load returns 512 bytes at
//                       128 a cycle).  Operands arrive by cp.async, 16 of K a step, four stages.  64 x 64
//                       tiles of two warps: 4096^3 5.69 -> 3.17 ms (43 TFLOP/s), 1129 x 1024 x 3072
//                       515 -> 217 us.  128 x 128 tiles gave 41 TFLOP/s and leave narrow outputs with too
//                       few blocks; packed pairs of FMAs need moves to double one operand and gave 40.
#include "common.cuh"

namespace ek {

constexpr int kRun = 64;              // products summed in one chain

// 8 values of a row from column k on (zeros from K on).  VEC: the 32 bytes are aligned and whole.
template <bool VEC>
__device__ __forceinline__ void load8(float (&v)[8], const float* row, int k, int K) {
  if (VEC) {
    if (k < K) {
      asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                   : "l"(row + k));
      return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = k + j < K ? row[k + j] : 0.f;
  }
}

// ------------------------------------------------------------------------------- few rows
// Columns a lane: every x value that it fetches serves them all.
__host__ __device__ constexpr int few_cols(int mr) { return mr == 1 ? 1 : mr <= 4 ? 2 : 4; }
__host__ __device__ constexpr int few_warps(int mr) { return mr <= 8 ? 8 : 4; }      // (the runs' sums fit 48 KB)

// MR rows (M <= MR).  Lane = 8 groups of columns x 4 runs; a warp takes 4 runs at a time.
template <int MR, bool VEC>
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
          for (int c = 0; c < CPL; ++c) load8<VEC>(w[c][i], w_row[c], k0 + 8 * (i0 + i), K);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
#pragma unroll
          for (int m = 0; m < MR; ++m) {
            float x[8];
            load8<VEC>(x, A + (size_t)min(m, M - 1) * lda, k0 + 8 * (i0 + i), K);
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
constexpr int kStepK = 16, kStepLd = kStepK + 4, kStages = 4;
__host__ __device__ constexpr int tile_smem(int bm, int bn) { return kStages * (bm + bn) * kStepLd * 4; }

// 8 x 8 outputs a thread: rows ty + i TY, columns tx + j TX.
template <int BM, int BN, bool VEC>
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
      if (VEC) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
        const int bytes = ok && k < K ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(bytes ? src + k : src), "r"(bytes)
                     : "memory");
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[j] = ok && k + j < K ? src[k + j] : 0.f;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
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
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();                           // the step's operands are there, and the stage refilled below is free
    if (s + kStages - 1 < steps) copy(s + kStages - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
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

template <int BM, int BN, bool VEC>
static int launch_tile(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc,
                       cudaStream_t stream) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return EK_ERR_ARG;
  auto kernel = sgemm_tile_kernel<BM, BN, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, tile_smem(BM, BN));
  if (e != cudaSuccess) return (int)e;
  kernel<<<grid, BM / 8 * (BN / 8), tile_smem(BM, BN), stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
  return (int)cudaGetLastError();
}

template <bool VEC>
static int launch_sgemm(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc,
                        cudaStream_t stream) {
  // 5 to 16 rows of many columns: x is read often enough for the few-row form to be bound by L1, and there
  // are columns enough for tiles (16 x 151936 x 1024: 425 us against 248; 12 x 40000 x 1024: 114 against 87;
  // but 16 x 6144 x 1024: 30 against 74)
  if (M <= 16 && !(M > 4 && N > 24576)) {
    const int mr = M == 1 ? 1 : M <= 4 ? 4 : M <= 8 ? 8 : 16;
    const int threads = 32 * min(few_warps(mr), (K + 4 * kRun - 1) / (4 * kRun));
    const dim3 grid((N + 8 * few_cols(mr) - 1) / (8 * few_cols(mr)));
    if (mr == 1) sgemm_few_rows_kernel<1, VEC><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    else if (mr == 4) sgemm_few_rows_kernel<4, VEC><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    else if (mr == 8) sgemm_few_rows_kernel<8, VEC><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    else sgemm_few_rows_kernel<16, VEC><<<grid, threads, 0, stream>>>(C, A, W, M, N, K, lda, ldw, ldc);
    return (int)cudaGetLastError();
  }
  if (M <= 16) return launch_tile<16, 128, VEC>(C, A, W, M, N, K, lda, ldw, ldc, stream);
  return launch_tile<64, 64, VEC>(C, A, W, M, N, K, lda, ldw, ldc, stream);
}

}  // namespace ek

EK_EXPORT int ek_gemm_nt_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda,
                             int ldw, int ldc, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldc < N) return EK_ERR_ARG;
  const bool vec = K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && ((uintptr_t)A & 31) == 0 && ((uintptr_t)W & 31) == 0;
  return vec ? ek::launch_sgemm<true>(C, A, W, M, N, K, lda, ldw, ldc, stream)
             : ek::launch_sgemm<false>(C, A, W, M, N, K, lda, ldw, ldc, stream);
}
