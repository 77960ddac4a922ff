// The gated delta rule over long stretches of tokens, 32 (kChunk) at a time (32-bit throughout).
//
// Token by token (delta.cu) a prompt is a chain of a matrix-vector product and an update per token.  Within a
// chunk of C tokens that starts from S, with the decays' products G(s, t) = g_(s+1) ... g_t per channel,
//     u_t = beta_t (v_t - k_t . G(0, t) S - sum_(s<t) A_ts u_s)        A_ts = k_t . G(s, t) k_s
//     o_t = q_t . G(0, t) S + sum_(s<=t) B_ts u_s                      B_ts = q_t . G(s, t) k_s
//     S'  = G(0, C) S + sum_s (G(s, C) k_s) u_s^T
// so with the lower triangular T = (1 + diag(beta) A)^-1 diag(beta), K~_t = G(0, t) k_t, Q~_t = G(0, t) q_t:
//     U = Y - W S,   O = Y' + Q' S       W = T K~,  Y = T V,  Q' = Q~ - B W,  Y' = B Y.
// Every G is a running product of decays: nothing is divided by a decay and no exponential is taken, so strong
// decays underflow to the zeros that they are token by token.  (That is also why A and B are built from running
// products instead of a matrix product of scaled keys.)
//
//   delta_chunk_prepare  W, Q', K^ = G(s, C) k, Y, Y' and G(0, C) of every chunk and head: all of them at once
//   delta_chunk_scan     the chain over the chunks: a block holds 16 columns of S of one head; a chunk is two
//                        small matrix products, [W ; Q'] S and K^T U, instead of 32 dependent steps
//
// Both are bound by the shared-memory reads and exchanges that feed the FMAs (a warp's 16-byte load takes four
// cycles; the scan with 512 threads instead of 256 took 235 us instead of 206).  Measured (2,048 tokens, 16 heads of
// 128 x 128, one prompt; the walk token by token takes 696 us): 106 + 206 us.  Errors against 64 bits: 1.6e-7 (o) and
// 1.4e-7 (S), 1.7e-7 and 1.6e-7 token by token.
#include "common.cuh"

namespace ek {

constexpr int kChunk = 32;
constexpr int kChunkCols = 16;               // columns of S a block of the scan holds
constexpr int kChunkThreads = 256;

struct ChunkShape {
  int heads, kv_heads, vdim;                 // (the key size is the kernels' D)
};

// Chunk `idx` of the step: which sequence, its first row, its rows, and its number among all chunks (or -1).
__device__ __forceinline__ int find_chunk(const int* cu_seqlens, int n_seqs, int idx, int& first, int& rows) {
  for (int b = 0; b < n_seqs; ++b) {
    const int n = cu_seqlens[b + 1] - cu_seqlens[b];
    const int chunks = (n + kChunk - 1) / kChunk;
    if (idx < chunks) {
      first = cu_seqlens[b] + idx * kChunk;
      rows = min(kChunk, n - idx * kChunk);
      return b;
    }
    idx -= chunks;
  }
  return -1;
}

template <int D>
__host__ __device__ constexpr int chunk_ld() { return D + 4; }
constexpr int kTriLd = kChunk + 4;

template <int D>
constexpr size_t chunk_prepare_smem(int vdim) {
  const int wide = vdim > D ? vdim : D;
  return sizeof(float) * (size_t)(4 * kChunk * chunk_ld<D>() + kChunk * (wide + 4) + 3 * kChunk * kTriLd + kChunk);
}

// acc[8][4] += L[8 rg + i][s] X[s][4 cg + c] over s < 8 rg + 8, L lower triangular and stored transposed
// (Lt[s][t]): the diagonal 8 x 8 piece takes only s <= t, so that a row meets nothing behind it.
__device__ __forceinline__ void tri_product(float (&acc)[8][4], const float* Lt, const float* X, int ldx, int rg, int cg) {
  auto step = [&](int s, int skip) {
    const float4 a0 = *reinterpret_cast<const float4*>(Lt + s * kTriLd + 8 * rg);
    const float4 a1 = *reinterpret_cast<const float4*>(Lt + s * kTriLd + 8 * rg + 4);
    const float4 x = *reinterpret_cast<const float4*>(X + s * ldx + 4 * cg);
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < skip) continue;
      acc[i][0] = fmaf(a[i], x.x, acc[i][0]);
      acc[i][1] = fmaf(a[i], x.y, acc[i][1]);
      acc[i][2] = fmaf(a[i], x.z, acc[i][2]);
      acc[i][3] = fmaf(a[i], x.w, acc[i][3]);
    }
  };
#pragma unroll 4
  for (int s = 0; s < 8 * rg; ++s) step(s, 0);
#pragma unroll
  for (int j = 0; j < 8; ++j) step(8 * rg + j, j);
}

// grid (chunks upper bound, heads).  qn, kn [T, kv_heads D]; v [T, heads vdim], overwritten by Y; decay [T, heads D]
// (or [T, heads] with decay_per_head); beta [T, heads].  Writes w, qp, kh [T, heads D] (kh may be `decay` itself),
// o [T, heads vdim] = Y', gam [chunk, heads, D].
template <int D>
__global__ void __launch_bounds__(kChunkThreads)
delta_chunk_prepare_kernel(float* __restrict__ w_out, float* __restrict__ qp_out, float* kh_out,
                           float* __restrict__ v, float* __restrict__ o, float* __restrict__ gam,
                           const float* __restrict__ qn, const float* __restrict__ kn, const float* decay,
                           const float* __restrict__ beta, const int* __restrict__ cu_seqlens, int n_seqs,
                           const int* __restrict__ positions, ChunkShape sh, int decay_per_head) {
  constexpr int LD = chunk_ld<D>();
  extern __shared__ __align__(16) float chunk_s[];
  const int wide = (sh.vdim > D ? sh.vdim : D) + 4;
  float* q_s = chunk_s;                        // [32][LD]: q, then Q~
  float* k_s = q_s + kChunk * LD;              // k
  float* g_s = k_s + kChunk * LD;              // decays
  float* y_s = k_s;                            // [32][wide] (wide <= 2 LD) over both, later: W, then Y
  float* t_s = g_s + kChunk * LD;              // K~
  float* v_s = t_s + kChunk * LD;              // [32][wide]: v
  float* a_s = v_s + kChunk * wide;            // [s][t]: A transposed
  float* b_s = a_s + kChunk * kTriLd;          // [s][t]: B transposed
  float* i_s = b_s + kChunk * kTriLd;          // [s][t]: T transposed
  float* beta_s = i_s + kChunk * kTriLd;
  __shared__ int where[3];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y;
  if (tid == 0) {
    int first = 0, rows = 0;
    where[2] = find_chunk(cu_seqlens, n_seqs, blockIdx.x, first, rows);
    where[0] = first; where[1] = rows;
  }
  __syncthreads();
  const int first = where[0], rows = where[1];
  if (where[2] < 0 || positions[first] < 0) return;
  const int kvh = h / (sh.heads / sh.kv_heads), E = sh.vdim;
  // tokens behind the last: k, q, v, beta 0 and decay 1 leave everything as it is
  for (int i = tid; i < kChunk * (D / 4); i += kChunkThreads) {
    const int t = i / (D / 4), c = i % (D / 4) * 4;
    const size_t row = first + t;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q, g = make_float4(1.f, 1.f, 1.f, 1.f);
    if (t < rows) {
      q = *reinterpret_cast<const float4*>(qn + (row * sh.kv_heads + kvh) * D + c);
      k = *reinterpret_cast<const float4*>(kn + (row * sh.kv_heads + kvh) * D + c);
      if (decay_per_head) {
        const float x = decay[row * sh.heads + h];
        g = make_float4(x, x, x, x);
      } else {
        g = *reinterpret_cast<const float4*>(decay + (row * sh.heads + h) * D + c);
      }
    }
    *reinterpret_cast<float4*>(q_s + t * LD + c) = q;
    *reinterpret_cast<float4*>(k_s + t * LD + c) = k;
    *reinterpret_cast<float4*>(g_s + t * LD + c) = g;
  }
  for (int i = tid; i < kChunk * (E / 4); i += kChunkThreads) {
    const int t = i / (E / 4), c = i % (E / 4) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < rows) x = *reinterpret_cast<const float4*>(v + ((size_t)(first + t) * sh.heads + h) * E + c);
    *reinterpret_cast<float4*>(v_s + t * wide + c) = x;
  }
  if (tid < kChunk) beta_s[tid] = tid < rows ? beta[(size_t)(first + tid) * sh.heads + h] : 0.f;
  for (int i = tid; i < kChunk * kTriLd; i += kChunkThreads) a_s[i] = b_s[i] = i_s[i] = 0.f;
  __syncthreads();

  // A and B: a warp takes two keys s at a time (2 w' and 2 w' + 1 for w' = warp and 15 - warp: equal shares), the
  // lanes their channels; the keys decay on the way to every later token t
  constexpr int PER = D / 32;                  // channels a lane (lane, lane + 32, ...)
#pragma unroll 1
  for (int round = 0; round < 2; ++round) {
    const int s0 = 2 * (round == 0 ? warp : 15 - warp);
    float x0[PER], x1[PER];
#pragma unroll
    for (int c = 0; c < PER; ++c) { x0[c] = k_s[s0 * LD + lane + 32 * c]; x1[c] = 0.f; }
#pragma unroll 1
    for (int t = s0; t < kChunk; ++t) {
      float r[4] = {0.f, 0.f, 0.f, 0.f};        // A_t,s0  B_t,s0  A_t,s0+1  B_t,s0+1
#pragma unroll
      for (int c = 0; c < PER; ++c) {
        const float g = g_s[t * LD + lane + 32 * c], k = k_s[t * LD + lane + 32 * c], q = q_s[t * LD + lane + 32 * c];
        if (t > s0) x0[c] *= g;
        x1[c] = t == s0 + 1 ? k : x1[c] * g;
        r[0] = fmaf(x0[c], k, r[0]);
        r[1] = fmaf(x0[c], q, r[1]);
        r[2] = fmaf(x1[c], k, r[2]);
        r[3] = fmaf(x1[c], q, r[3]);
      }
      // sums over the lanes, each value ending with a quarter of them
      const bool hi = lane & 16, mid = lane & 8;
      const float e0 = __shfl_xor_sync(0xffffffffu, hi ? r[0] : r[2], 16), e1 = __shfl_xor_sync(0xffffffffu, hi ? r[1] : r[3], 16);
      const float a0 = (hi ? r[2] : r[0]) + e0, a1 = (hi ? r[3] : r[1]) + e1;
      float z = (mid ? a1 : a0) + __shfl_xor_sync(0xffffffffu, mid ? a0 : a1, 8);
      z += __shfl_xor_sync(0xffffffffu, z, 4);
      z += __shfl_xor_sync(0xffffffffu, z, 2);
      z += __shfl_xor_sync(0xffffffffu, z, 1);
      const int s = s0 + (hi ? 1 : 0);
      if ((lane & 7) == 0 && t >= s) {
        if (mid) b_s[s * kTriLd + t] = z;
        else if (t > s) a_s[s * kTriLd + t] = z;
      }
    }
  }
  // running products: K~ and Q~ from the front, K^ from the back
  __syncthreads();
  if (tid < D) {
    float f = 1.f;
    for (int t = 0; t < kChunk; ++t) {
      f *= g_s[t * LD + tid];
      t_s[t * LD + tid] = k_s[t * LD + tid] * f;
      q_s[t * LD + tid] *= f;
    }
    gam[((size_t)blockIdx.x * sh.heads + h) * D + tid] = f;
  }
  if (tid >= kChunkThreads - D) {
    const int c = tid - (kChunkThreads - D);
    float f = 1.f;
    for (int s = kChunk - 1; s >= 0; --s) {
      if (s < rows) kh_out[((size_t)(first + s) * sh.heads + h) * D + c] = k_s[s * LD + c] * f;
      f *= g_s[s * LD + c];
    }
  }
  // T by forward substitution: lane j of the first warp its column j
  if (warp == 0) {
    float col[kChunk];
#pragma unroll
    for (int t = 0; t < kChunk; ++t) {
      float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < t; ++s) p[s & 3] = fmaf(a_s[s * kTriLd + t], col[s], p[s & 3]);
      const float b = beta_s[t];
      col[t] = t < lane ? 0.f : t == lane ? b : -b * ((p[0] + p[1]) + (p[2] + p[3]));
      i_s[lane * kTriLd + t] = col[t];
    }
  }
  __syncthreads();

  // W = T K~ (kept in shared memory for Q' = Q~ - B W)
  const int rg = tid / 64, cg = tid % 64;       // 8 rows, 4 columns of up to 256
  for (int c = cg; c < D / 4; c += 64) {
    float acc[8][4] = {};
    tri_product(acc, i_s, t_s, LD, rg, c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = 8 * rg + i;
      const float4 x = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(y_s + t * wide + 4 * c) = x;
      if (t < rows) *reinterpret_cast<float4*>(w_out + ((size_t)(first + t) * sh.heads + h) * D + 4 * c) = x;
    }
  }
  __syncthreads();
  for (int c = cg; c < D / 4; c += 64) {
    float acc[8][4] = {};
    tri_product(acc, b_s, y_s, wide, rg, c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = 8 * rg + i;
      if (t >= rows) continue;
      const float4 q = *reinterpret_cast<const float4*>(q_s + t * LD + 4 * c);
      *reinterpret_cast<float4*>(qp_out + ((size_t)(first + t) * sh.heads + h) * D + 4 * c) =
          make_float4(q.x - acc[i][0], q.y - acc[i][1], q.z - acc[i][2], q.w - acc[i][3]);
    }
  }
  __syncthreads();
  // Y = T V and Y' = B Y
  for (int c = cg; c < E / 4; c += 64) {
    float acc[8][4] = {};
    tri_product(acc, i_s, v_s, wide, rg, c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = 8 * rg + i;
      const float4 x = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(y_s + t * wide + 4 * c) = x;
      if (t < rows) *reinterpret_cast<float4*>(v + ((size_t)(first + t) * sh.heads + h) * E + 4 * c) = x;
    }
  }
  __syncthreads();
  for (int c = cg; c < E / 4; c += 64) {
    float acc[8][4] = {};
    tri_product(acc, b_s, y_s, wide, rg, c);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = 8 * rg + i;
      if (t < rows)
        *reinterpret_cast<float4*>(o + ((size_t)(first + t) * sh.heads + h) * E + 4 * c) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
  }
}

template <int D>
__host__ __device__ constexpr size_t chunk_scan_smem() {
  // S, two buffers of W, Q', K^ and of Y, Y', U
  return sizeof(float) * (size_t)(kChunkCols * chunk_ld<D>() + 2 * 3 * kChunk * chunk_ld<D>() +
                                  (2 * 2 + 1) * kChunk * kChunkCols + 2 * D);
}

// a block per (sequence, head, tile of 16 columns), tiles fastest.
template <int D>
__global__ void __launch_bounds__(kChunkThreads)
delta_chunk_scan_kernel(float* __restrict__ o, const float* __restrict__ w, const float* __restrict__ qp,
                        const float* __restrict__ kh, const float* __restrict__ y, const float* __restrict__ gam,
                        float* __restrict__ state, size_t slot_stride, const int* __restrict__ cu_seqlens,
                        const int* __restrict__ positions, const int* __restrict__ token_slot, ChunkShape sh) {
  constexpr int LD = chunk_ld<D>(), PIECES = D / 4;
  constexpr int BUF = 3 * kChunk * LD;
  extern __shared__ __align__(16) float chunk_s[];
  float* s_s = chunk_s;                        // [16 columns][LD]
  float* ops = s_s + kChunkCols * LD;          // [2][W | Q' | K^][32][LD]
  float* ys = ops + 2 * BUF;                   // [2][Y | Y'][32][16]
  float* u_s = ys + 2 * 2 * kChunk * kChunkCols;      // [32][16]
  float* gam_s = u_s + kChunk * kChunkCols;    // [2][D]
  pdl_launch_dependents();
  pdl_wait();
  // sequences slowest, so that the blocks of the longest one spread over the SMs
  const int tiles = (sh.vdim + kChunkCols - 1) / kChunkCols, tile = blockIdx.x % tiles;
  const int tid = threadIdx.x, b = blockIdx.x / tiles / sh.heads, h = blockIdx.x / tiles % sh.heads;
  const int start = cu_seqlens[b], n = cu_seqlens[b + 1] - start;
  if (n <= 0 || positions[start] < 0) return;
  int chunk0 = 0;                              // the sequence's first chunk among all
  for (int i = 0; i < b; ++i) chunk0 += (cu_seqlens[i + 1] - cu_seqlens[i] + kChunk - 1) / kChunk;
  const int E = sh.vdim, col0 = tile * kChunkCols, cols = min(kChunkCols, E - col0);
  float* S = state + (size_t)token_slot[start] * slot_stride + ((size_t)h * E + col0) * D;

  auto copy16 = [&](float* dst, const float* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
  };
  auto fetch = [&](int c0, int buf) {          // chunk c0 .. of the sequence; zeros behind its last token
    const int rows = min(kChunk, n - c0);
    float* to = ops + buf * BUF;
#pragma unroll
    for (int i = tid; i < 3 * kChunk * PIECES; i += kChunkThreads) {
      const int which = i / (kChunk * PIECES), t = i / PIECES % kChunk, c = i % PIECES * 4;
      const float* src = which == 0 ? w : which == 1 ? qp : kh;
      const bool ok = t < rows;
      copy16(to + (which * kChunk + t) * LD + c, src + ((size_t)(start + c0 + (ok ? t : 0)) * sh.heads + h) * D + c, ok);
    }
    {
      const int which = tid / 128, t = tid % 128 / 4, c = tid % 4 * 4;       // 2 x 32 x 4 pieces: one a thread
      const bool ok = t < rows && c < cols;
      copy16(ys + ((buf * 2 + which) * kChunk + t) * kChunkCols + c,
             (which ? o : y) + ((size_t)(start + c0 + (t < rows ? t : 0)) * sh.heads + h) * E + col0 + (c < cols ? c : 0), ok);
    }
    if (tid < PIECES)
      copy16(gam_s + buf * D + tid * 4, gam + ((size_t)(chunk0 + c0 / kChunk) * sh.heads + h) * D + tid * 4, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, 0);
  for (int i = tid; i < kChunkCols * PIECES; i += kChunkThreads) {
    const int c = i / PIECES, d = i % PIECES * 4;
    const float4 x = c < cols ? *reinterpret_cast<const float4*>(S + (size_t)c * D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(s_s + c * LD + d) = x;
  }

  // first product: rows ra + 8 i of [W ; Q'] (64), columns ca + 4 j, dimensions 4 (part + 8 m): eight lanes share a sum
  const int part = tid & 7, ca = (tid >> 3) & 3, ra = tid >> 5;
  // second: dimensions 4 dg .. + 3, columns 4 cb .. + 3, tokens of one parity: two lanes share a sum
  constexpr int DG = D / 4;
  const int half = tid & 1, cb = (tid >> 1) & 3, dg = tid >> 3;

  int buf = 0;
  for (int c0 = 0; c0 < n; c0 += kChunk, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                           // the chunk's operands and S are there; the other buffer is free
    if (c0 + kChunk < n) fetch(c0 + kChunk, buf ^ 1);
    const float* wq = ops + buf * BUF;
    {
      float acc[8][4] = {};
#pragma unroll
      for (int m = 0; m < D / 32; ++m) {
        const int d = 4 * (part + 8 * m);
        float4 s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = *reinterpret_cast<const float4*>(s_s + (ca + 4 * j) * LD + d);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 x = *reinterpret_cast<const float4*>(wq + (ra + 8 * i) * LD + d);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[i][j] = fmaf(x.w, s[j].w, fmaf(x.z, s[j].z, fmaf(x.y, s[j].y, fmaf(x.x, s[j].x, acc[i][j]))));
        }
      }
      // sums over the eight lanes: a lane ends with the row ra + 8 part (its bits choose halves)
      float r4[4][4], r2[2][4], r1[4];
      const bool p4 = part & 4, p2 = part & 2, p1 = part & 1;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          r4[i][j] = (p4 ? acc[4 + i][j] : acc[i][j]) + __shfl_xor_sync(0xffffffffu, p4 ? acc[i][j] : acc[4 + i][j], 4);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          r2[i][j] = (p2 ? r4[2 + i][j] : r4[i][j]) + __shfl_xor_sync(0xffffffffu, p2 ? r4[i][j] : r4[2 + i][j], 2);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        r1[j] = (p1 ? r2[1][j] : r2[0][j]) + __shfl_xor_sync(0xffffffffu, p1 ? r2[0][j] : r2[1][j], 1);
      const int row = ra + 8 * part;           // 0 .. 31: W's, 32 .. 63: Q's
      if (row < kChunk) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          u_s[row * kChunkCols + ca + 4 * j] = ys[(buf * 2 * kChunk + row) * kChunkCols + ca + 4 * j] - r1[j];
      } else {
        const int t = row - kChunk;
        if (c0 + t < n) {
          float* to = o + ((size_t)(start + c0 + t) * sh.heads + h) * E + col0;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (ca + 4 * j < cols) to[ca + 4 * j] = ys[((buf * 2 + 1) * kChunk + t) * kChunkCols + ca + 4 * j] + r1[j];
        }
      }
    }
    __syncthreads();                           // U is there; S has been read
    const float* k = wq + 2 * kChunk * LD;
    if (dg < DG) {
      float acc[4][4] = {};
#pragma unroll 8
      for (int t = half; t < kChunk; t += 2) {
        const float4 x = *reinterpret_cast<const float4*>(k + t * LD + 4 * dg);
        const float4 u = *reinterpret_cast<const float4*>(u_s + t * kChunkCols + 4 * cb);
        const float xv[4] = {x.x, x.y, x.z, x.w}, uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[c][i] = fmaf(xv[i], uv[c], acc[c][i]);
      }
      const float4 f = *reinterpret_cast<const float4*>(gam_s + buf * D + 4 * dg);
#pragma unroll
      for (int c = 0; c < 2; ++c) {            // the even lane ends with columns 0, 1 of its four, the odd one with 2, 3
        float z[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          z[i] = (half ? acc[2 + c][i] : acc[c][i]) + __shfl_xor_sync(0xffffffffu, half ? acc[c][i] : acc[2 + c][i], 1);
        float4* at = reinterpret_cast<float4*>(s_s + (4 * cb + 2 * half + c) * LD + 4 * dg);
        const float4 s = *at;
        *at = make_float4(fmaf(f.x, s.x, z[0]), fmaf(f.y, s.y, z[1]), fmaf(f.z, s.z, z[2]), fmaf(f.w, s.w, z[3]));
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < cols * PIECES; i += kChunkThreads) {
    const int c = i / PIECES, d = i % PIECES * 4;
    *reinterpret_cast<float4*>(S + (size_t)c * D + d) = *reinterpret_cast<const float4*>(s_s + c * LD + d);
  }
}

template <int D>
static int launch_chunks(float* o, float* w, float* qp, float* kh, float* v, float* gam, const float* qn, const float* kn,
                         const float* decay, const float* beta, float* state, size_t slot_stride, const int* cu_seqlens,
                         const int* positions, const int* token_slot, int n_seqs, int chunks, ChunkShape sh,
                         int decay_per_head, cudaStream_t stream) {
  const size_t smem = chunk_prepare_smem<D>(sh.vdim);
  auto prepare = delta_chunk_prepare_kernel<D>;
  auto scan = delta_chunk_scan_kernel<D>;
  cudaError_t e = cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chunk_scan_smem<D>());
  if (e != cudaSuccess) return (int)e;
  e = launch_pdl(prepare, dim3(chunks, sh.heads), dim3(kChunkThreads), smem, stream, w, qp, kh, v, o, gam, qn, kn, decay,
                 beta, cu_seqlens, n_seqs, positions, sh, decay_per_head);
  if (e != cudaSuccess) return (int)e;
  const long long blocks = (long long)n_seqs * sh.heads * ((sh.vdim + kChunkCols - 1) / kChunkCols);
  if (blocks > 0x7fffffffLL || sh.heads > 65535 || sh.vdim > 65535 * kChunkCols) return EK_ERR_ARG;
  return (int)launch_pdl(scan, dim3((unsigned)blocks), dim3(kChunkThreads),
                         chunk_scan_smem<D>(), stream, o, w, qp, kh, v, gam, state, slot_stride, cu_seqlens, positions,
                         token_slot, sh);
}

}  // namespace ek

// The recurrence of ek_delta_scan for key sizes 64 and 128 and value sizes in steps of 4 up to twice that, by chunks.
// `v` [T, heads vdim] is overwritten; `decay` too, unless `kh` is memory of its own (decay_per_head needs that).
// w, qp, kh: [T, heads dim] of scratch; gam: [chunks, heads, dim], chunks = the sequences' tokens / 32 rounded up, summed.
EK_EXPORT int ek_delta_chunks(float* o, const float* qn, const float* kn, float* v, const float* beta, const float* decay,
                              float* w, float* qp, float* kh, float* gam, float* state, long long slot_stride,
                              const int* cu_seqlens, const int* positions, const int* token_slot, int n_seqs, int chunks,
                              int heads, int kv_heads, int dim, int vdim, int decay_per_head, cudaStream_t stream) {
  using namespace ek;
  if (n_seqs <= 0 || chunks <= 0) return 0;
  if (heads <= 0 || heads > 65535 || kv_heads <= 0 || heads % kv_heads || vdim <= 0 || vdim % 4 || vdim > 2 * dim ||
      slot_stride % 4 || (decay_per_head && kh == decay) ||
      (((uintptr_t)o | (uintptr_t)qn | (uintptr_t)kn | (uintptr_t)v | (uintptr_t)decay | (uintptr_t)w | (uintptr_t)qp |
        (uintptr_t)kh | (uintptr_t)gam | (uintptr_t)state) & 15))
    return EK_ERR_ARG;
  const ChunkShape sh{heads, kv_heads, vdim};
  if (dim == 128)
    return launch_chunks<128>(o, w, qp, kh, v, gam, qn, kn, decay, beta, state, (size_t)slot_stride, cu_seqlens, positions,
                              token_slot, n_seqs, chunks, sh, decay_per_head, stream);
  if (dim == 64)
    return launch_chunks<64>(o, w, qp, kh, v, gam, qn, kn, decay, beta, state, (size_t)slot_stride, cu_seqlens, positions,
                             token_slot, n_seqs, chunks, sh, decay_per_head, stream);
  return EK_ERR_ARG;
}
