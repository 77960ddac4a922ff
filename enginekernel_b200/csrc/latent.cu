// Latent attention: what stands between the projections and the attention kernels.
//
// A token's keys and values of all heads are functions of one latent vector c (size C) and one
// rotated key part r (size R) shared by the heads:  k_h = [W_uk,h c ; r],  v_h = W_uv,h c.  Only
// [c ; r] is cached, one row of D >= C + R values per token (padded with zeros to the row length
// the attention kernels take), and attention runs in the absorbed form
//     score_h(i, j) = (W_uk,h^T q_h,flat)(i) . c(j) + q_h,rot(i) . r(j),
//     out_h(i)      = W_uv,h sum_j p_h(i, j) c(j),
// that is: attention with ONE key head whose keys and values are both the cached rows, H query
// heads of size D, followed by a product per head.  Two kernels:
//   latent_prepare   norms of the two latents (32-bit), rotation of r, cache write, per token
//   head_linear      out[t, h, :] = W_h in[t, h, :] per head: the value up-projection, and - with the
//                    rotated tail - the absorbed query [W_uk,h^T q_h,flat ; rot(q_h,rot) ; 0]
// Norms, angles and rotations are computed in 32-bit; T is the activation / cache type.
#include <type_traits>

#include "common.cuh"

namespace ek {

// One block per token.  proj[t] = [dq (QR) | dkv latent (C) | key rot part (R)] in 32-bit.
//   cq[t, :QR]   = gain_q  * dq / rms(dq)                      (type T, feeds the q up-projection)
//                  or, without gain_q, the QR values as they are (a design whose queries - and whatever else
//                  reads the input beside them - are plain projections); QR = 0: there is no such part
//   page row     = [gain_kv * lat / rms(lat) | rot(r) | 0..]   (type T, D values)
// cos/sin: [positions, rot_dims / 2] in 32-bit (any factor on them is already in the tables);
// dimension i < rot_dims/2 of r turns with dimension i + rot_dims/2, the rest of r passes.
//
// What bounds it, with few tokens, is the chain of loads that wait for one another.  The gains are fetched before the wait
// for the kernel ahead; behind it the row comes into registers while the token's place and its angles are looked up, and
// both norms are one reduction.  (Positions stand behind the wait: ahead of it an ordinary load may find the step before's,
// see common.cuh, and reading them there gained nothing.)
// 8 tokens of 768 + 192 + 64 values in a captured step: 6.2 us with every load in its place, now 2.1.
constexpr int kPrepKeep = 8;         // values of the first part a thread keeps, and of the latent a quarter of that
template <typename T>
__global__ void latent_prepare_kernel(T* __restrict__ cq, const float* __restrict__ proj, int proj_stride,
                                      const float* __restrict__ gain_q, const float* __restrict__ gain_kv,
                                      float eps, const float* __restrict__ cos_t,
                                      const float* __restrict__ sin_t, int rot_dims,
                                      const int* __restrict__ positions, const int* __restrict__ token_slot,
                                      T* __restrict__ pages, const int* __restrict__ block_table,
                                      int table_stride, int QR, int C, int R, int D, int write_cache) {
  constexpr int KEEP_C = kPrepKeep / 4;
  __shared__ float scratch[2][32];
  pdl_launch_dependents();
  const int t = blockIdx.x, tid = threadIdx.x, threads = blockDim.x;
  const int half = rot_dims / 2;
  float gq[kPrepKeep], gk[KEEP_C], c0 = 1.f, s0 = 0.f;
#pragma unroll
  for (int j = 0; j < kPrepKeep; ++j) gq[j] = gain_q != nullptr && tid + j * threads < QR ? gain_q[tid + j * threads] : 1.f;
#pragma unroll
  for (int j = 0; j < KEEP_C; ++j) gk[j] = write_cache && tid + j * threads < C ? gain_kv[tid + j * threads] : 0.f;
  pdl_wait();
  const int pos = positions[t];
  const int slot = token_slot[t];
  const float* row = proj + (size_t)t * proj_stride;
  const float* lat = row + QR;
  const float* r = lat + C;
  float rq[kPrepKeep], rk[KEEP_C], r0 = 0.f, r1 = 0.f;
#pragma unroll
  for (int j = 0; j < kPrepKeep; ++j) rq[j] = tid + j * threads < QR ? row[tid + j * threads] : 0.f;
  const bool cached = write_cache && pos >= 0;    // (uniform over the block)
  float sums[2] = {0.f, 0.f};
  T* dst = nullptr;
  if (cached) {
    const int page = block_table[(size_t)slot * table_stride + pos / EK_PAGE];
    dst = pages + ((size_t)page * EK_PAGE + (pos & (EK_PAGE - 1))) * (size_t)D;
    if (tid < rot_dims) {
      const size_t at = (size_t)pos * half + (tid < half ? tid : tid - half);
      c0 = cos_t[at];
      s0 = sin_t[at];
    }
#pragma unroll
    for (int j = 0; j < KEEP_C; ++j) rk[j] = tid + j * threads < C ? lat[tid + j * threads] : 0.f;
    if (tid < R) r0 = r[tid];
    if (tid < rot_dims) r1 = r[tid < half ? tid + half : tid - half];
#pragma unroll
    for (int j = 0; j < KEEP_C; ++j) sums[1] += rk[j] * rk[j];
    for (int i = tid + KEEP_C * threads; i < C; i += threads) sums[1] += lat[i] * lat[i];
  }
  if (gain_q != nullptr) {
#pragma unroll
    for (int j = 0; j < kPrepKeep; ++j) sums[0] += rq[j] * rq[j];
    for (int i = tid + kPrepKeep * threads; i < QR; i += threads) sums[0] += row[i] * row[i];
  }
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    sums[w] = warp_sum(sums[w]);
    if ((tid & 31) == 0) scratch[w][tid >> 5] = sums[w];
  }
  __syncthreads();
  sums[0] = sums[1] = 0.f;
  for (int w = 0; w < threads / 32; ++w) {
    sums[0] += scratch[0][w];
    sums[1] += scratch[1][w];
  }
  const float inv_q = gain_q != nullptr ? rsqrtf(sums[0] / (float)QR + eps) : 1.f;
  T* q = cq + (size_t)t * QR;
#pragma unroll
  for (int j = 0; j < kPrepKeep; ++j)
    if (tid + j * threads < QR) q[tid + j * threads] = from_f<T>(gain_q != nullptr ? rq[j] * inv_q * gq[j] : rq[j]);
  for (int i = tid + kPrepKeep * threads; i < QR; i += threads)
    q[i] = from_f<T>(gain_q != nullptr ? row[i] * inv_q * gain_q[i] : row[i]);

  if (!cached) return;
  const float inv_k = rsqrtf(sums[1] / (float)C + eps);
#pragma unroll
  for (int j = 0; j < KEEP_C; ++j)
    if (tid + j * threads < C) dst[tid + j * threads] = from_f<T>(rk[j] * inv_k * gk[j]);
  for (int i = tid + KEEP_C * threads; i < C; i += threads) dst[i] = from_f<T>(lat[i] * inv_k * gain_kv[i]);
  if (tid < R) dst[C + tid] = from_f<T>(tid >= rot_dims ? r0 : tid < half ? r0 * c0 - r1 * s0 : r0 * c0 + r1 * s0);
  for (int i = tid + threads; i < R; i += threads) {
    float v = r[i];
    if (i < half) {
      const float c = cos_t[(size_t)pos * half + i], s = sin_t[(size_t)pos * half + i];
      v = r[i] * c - r[i + half] * s;
    } else if (i < rot_dims) {
      const float c = cos_t[(size_t)pos * half + i - half], s = sin_t[(size_t)pos * half + i - half];
      v = r[i] * c + r[i - half] * s;
    }
    dst[C + i] = from_f<T>(v);
  }
  for (int i = C + R + tid; i < D; i += threads) dst[i] = from_f<T>(0.f);
}

constexpr int kHeadTokens = 8;       // tokens a block of the per-head products takes
constexpr int kHeadOuts = 32;        // output values a block takes ...
constexpr int kHeadSlices = 4;       // ... each summed by this many threads over a quarter of the inputs
constexpr int kHeadThreads = kHeadOuts * kHeadSlices;

// out[t, h, o] = sum_i w[h, i, o] * in[t, h, i]   for o < n_out, i < n_in.
// w is laid out [heads, n_in, n_out] (neighbouring threads read neighbouring weights).  grid (token tiles, heads, output tiles of 32); a warp takes a quarter of the
// inputs for the tile's 32 outputs and the four warps' sums meet in shared memory, so that with few
// tokens the chain of loads is short and the weights are spread over many blocks.  If rot_dims >= 0
// the block with blockIdx.z == 0 also writes the rotated tail: out[t, h, n_out + i] =
// rot(in[t, h, n_in + i]) for i < R and zeros up to out_head_stride (the absorbed query).
template <typename T>
__global__ void __launch_bounds__(kHeadThreads)
head_linear_kernel(T* __restrict__ out, int out_row_stride, int out_head_stride,
                   const T* __restrict__ in, int in_row_stride, int in_head_stride,
                   const T* __restrict__ w, int n_tokens, int n_in, int n_out, int R, int rot_dims,
                   const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                   const int* __restrict__ positions) {
  extern __shared__ float in_s[];               // [kHeadTokens][n_in + R]
  __shared__ float part_s[kHeadSlices][kHeadTokens][kHeadOuts];
  pdl_launch_dependents();
  const int t0 = blockIdx.x * kHeadTokens, h = blockIdx.y, tid = threadIdx.x;
  const int slice = tid / kHeadOuts, oo = tid % kHeadOuts;
  const int o = blockIdx.z * kHeadOuts + oo;
  const int per = (n_in + kHeadSlices - 1) / kHeadSlices;
  const int i0 = slice * per, i1 = min(n_in, i0 + per);
  const T* wp = o < n_out ? w + (size_t)h * n_in * n_out + o : nullptr;
  pdl_wait();
  const int nt = min(kHeadTokens, n_tokens - t0);
  const int width = n_in + (rot_dims >= 0 ? R : 0);
  for (int idx = tid; idx < kHeadTokens * width; idx += kHeadThreads) {
    const int tt = idx / width, i = idx % width;
    in_s[idx] = tt < nt ? to_f<T>(in[(size_t)(t0 + tt) * in_row_stride + (size_t)h * in_head_stride + i]) : 0.f;
  }
  __syncthreads();
  {
    float acc[kHeadTokens];
#pragma unroll
    for (int tt = 0; tt < kHeadTokens; ++tt) acc[tt] = 0.f;
    if (wp != nullptr) {
#pragma unroll 8
      for (int i = i0; i < i1; ++i) {
        const float wv = to_f<T>(wp[(size_t)i * n_out]);
#pragma unroll
        for (int tt = 0; tt < kHeadTokens; ++tt) acc[tt] = fmaf(wv, in_s[tt * width + i], acc[tt]);
      }
    }
#pragma unroll
    for (int tt = 0; tt < kHeadTokens; ++tt) part_s[slice][tt][oo] = acc[tt];
    __syncthreads();
    for (int idx = tid; idx < nt * kHeadOuts; idx += kHeadThreads) {
      const int tt = idx / kHeadOuts, o2 = blockIdx.z * kHeadOuts + idx % kHeadOuts;
      if (o2 < n_out) {
        float v = 0.f;
#pragma unroll
        for (int sl = 0; sl < kHeadSlices; ++sl) v += part_s[sl][tt][idx % kHeadOuts];
        out[(size_t)(t0 + tt) * out_row_stride + (size_t)h * out_head_stride + o2] = from_f<T>(v);
      }
    }
  }
  if (rot_dims >= 0 && blockIdx.z == 0) {
    const int half = rot_dims / 2;
    const int tail = out_head_stride - n_out;
    for (int idx = tid; idx < nt * tail; idx += kHeadThreads) {
      const int tt = idx / tail, i = idx % tail;
      float v = 0.f;
      if (i < R) {
        const float* r = in_s + tt * width + n_in;
        const int pos = max(positions[t0 + tt], 0);
        v = r[i];
        if (i < half) {
          const float c = cos_t[(size_t)pos * half + i], s = sin_t[(size_t)pos * half + i];
          v = r[i] * c - r[i + half] * s;
        } else if (i < rot_dims) {
          const float c = cos_t[(size_t)pos * half + i - half], s = sin_t[(size_t)pos * half + i - half];
          v = r[i] * c + r[i - half] * s;
        }
      }
      out[(size_t)(t0 + tt) * out_row_stride + (size_t)h * out_head_stride + n_out + i] = from_f<T>(v);
    }
  }
}

// The rotated tail alone (no product), a block a token over all heads: 2,048 tokens of 16 heads of 64 values took the
// product's kernel, which also fetched the 128 values before each tail, 25 us, and take this one 9.
template <typename T>
__global__ void __launch_bounds__(256)
head_tail_kernel(T* __restrict__ out, int out_row_stride, int out_head_stride, const T* __restrict__ in, int in_row_stride,
                 int in_head_stride, int heads, int n_in, int n_out, int R, int rot_dims, const float* __restrict__ cos_t,
                 const float* __restrict__ sin_t, const int* __restrict__ positions) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, half = rot_dims / 2, tail = out_head_stride - n_out;
  const int pos = max(positions[t], 0);
  for (int idx = threadIdx.x; idx < heads * tail; idx += blockDim.x) {
    const int h = idx / tail, i = idx % tail;
    const T* r = in + (size_t)t * in_row_stride + (size_t)h * in_head_stride + n_in;
    float v = 0.f;
    if (i < R) {
      v = to_f<T>(r[i]);
      if (i < rot_dims) {
        const int j = i < half ? i : i - half;
        const float c = cos_t[(size_t)pos * half + j], s = sin_t[(size_t)pos * half + j];
        v = i < half ? v * c - to_f<T>(r[i + half]) * s : v * c + to_f<T>(r[j]) * s;
      }
    }
    out[(size_t)t * out_row_stride + (size_t)h * out_head_stride + n_out + i] = from_f<T>(v);
  }
}

// The same product in bfloat16 on mma.sync.m16n8k16 with the output values as the 16 rows and the tokens as the 8 columns,
// 32-bit sums.  With few tokens the weights are the work and latency bounds it: a block's weights [n_in][32] come by
// cp.async BEFORE the wait for the kernel ahead (they do not depend on it), a warp takes every fourth step of 16 inputs,
// and the four sums meet in shared memory.  The rotated tail, a chain of three loads, has a block of its own
// (blockIdx.z past the output tiles).  8 tokens of 16 heads in a captured step, 128 -> 192 with a tail and 192 -> 128:
// 10.0 and 6.8 us by the kernel above, 4.1 and 2.6 by this one.
constexpr int kHeadWRow = 2 * kHeadOuts + 16;    // bytes of a row of weights in shared memory: eight rows, eight bank groups
__host__ __device__ constexpr size_t head_mma_smem(int n_in) {
  return (size_t)n_in * kHeadWRow + (size_t)kHeadTokens * (2 * n_in + 16);
}
__global__ void __launch_bounds__(kHeadThreads)
head_linear_mma_kernel(bf16* __restrict__ out, int out_row_stride, int out_head_stride, const bf16* __restrict__ in,
                       int in_row_stride, int in_head_stride, const bf16* __restrict__ w, int n_tokens, int n_in, int n_out,
                       int R, int rot_dims, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                       const int* __restrict__ positions) {
  extern __shared__ __align__(16) unsigned char head_smem[];
  __shared__ float part_s[kHeadSlices][kHeadTokens][kHeadOuts + 1];
  pdl_launch_dependents();
  const int t0 = blockIdx.x * kHeadTokens, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = min(kHeadTokens, n_tokens - t0);
  const int o0 = blockIdx.z * kHeadOuts;
  if (o0 >= n_out) {                             // the tail's block
    pdl_wait();
    const int half = rot_dims / 2, tail = out_head_stride - n_out;
    for (int idx = tid; idx < nt * tail; idx += kHeadThreads) {
      const int tt = idx / tail, i = idx % tail;
      const bf16* r = in + (size_t)(t0 + tt) * in_row_stride + (size_t)h * in_head_stride + n_in;
      float v = 0.f;
      if (i < R) {
        v = to_f<bf16>(r[i]);
        if (i < rot_dims) {
          const float other = to_f<bf16>(r[i < half ? i + half : i - half]);
          const size_t at = (size_t)max(positions[t0 + tt], 0) * half + (i < half ? i : i - half);
          const float c = cos_t[at], s = sin_t[at];
          v = i < half ? v * c - other * s : v * c + other * s;
        }
      }
      out[(size_t)(t0 + tt) * out_row_stride + (size_t)h * out_head_stride + n_out + i] = from_f<bf16>(v);
    }
    return;
  }
  const int wide = min(kHeadOuts, n_out - o0) / 8;               // 16-byte pieces of a weight row that there are
  const uint32_t w_s = (uint32_t)__cvta_generic_to_shared(head_smem);
  unsigned char* in_s = head_smem + (size_t)n_in * kHeadWRow;
  const int in_bytes = 2 * n_in + 16;
  const bf16* wp = w + (size_t)h * n_in * n_out + o0;
  for (int idx = tid; idx < n_in * (kHeadOuts / 8); idx += kHeadThreads) {
    const int i = idx / (kHeadOuts / 8), c = idx % (kHeadOuts / 8);
    const int there = c < wide ? 16 : 0;                         // (a piece past the head's outputs is zeros)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(w_s + i * kHeadWRow + 16 * c),
                 "l"(wp + (size_t)i * n_out + (there ? 8 * c : 0)), "r"(there) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  pdl_wait();
  for (int idx = tid; idx < kHeadTokens * (n_in / 8); idx += kHeadThreads) {
    const int tt = idx / (n_in / 8), c = idx % (n_in / 8);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (tt < nt) v = *reinterpret_cast<const uint4*>(in + (size_t)(t0 + tt) * in_row_stride + (size_t)h * in_head_stride + 8 * c);
    *reinterpret_cast<uint4*>(in_s + tt * in_bytes + 16 * c) = v;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
  const int g = lane >> 2, tq = lane & 3;
  for (int k = 16 * warp; k < n_in; k += 16 * kHeadSlices) {
    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(in_s + g * in_bytes + 2 * (k + 2 * tq));
    const uint32_t b1 = *reinterpret_cast<const uint32_t*>(in_s + g * in_bytes + 2 * (k + 8 + 2 * tq));
    const uint32_t row = w_s + (k + (lane & 7) + 8 * (lane >> 4)) * kHeadWRow + 16 * ((lane >> 3) & 1);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      uint32_t a0, a1, a2, a3;
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3) : "r"(row + 32 * m) : "memory");
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(acc[m][0]), "+f"(acc[m][1]), "+f"(acc[m][2]), "+f"(acc[m][3])
                   : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) part_s[warp][2 * tq + (e & 1)][16 * m + g + 8 * (e >> 1)] = acc[m][e];
  __syncthreads();
  for (int idx = tid; idx < nt * kHeadOuts; idx += kHeadThreads) {
    const int tt = idx / kHeadOuts, o = idx % kHeadOuts;
    if (o0 + o >= n_out) continue;
    float v = 0.f;
#pragma unroll
    for (int sl = 0; sl < kHeadSlices; ++sl) v += part_s[sl][tt][o];
    out[(size_t)(t0 + tt) * out_row_stride + (size_t)h * out_head_stride + o0 + o] = from_f<bf16>(v);
  }
}

template <typename T>
static int launch_head_linear(T* out, int out_row_stride, int out_head_stride, const T* in,
                              int in_row_stride, int in_head_stride, const T* w, int n_tokens,
                              int heads, int n_in, int n_out, int R, int rot_dims, const float* cos_t,
                              const float* sin_t, const int* positions, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (heads <= 0 || heads > 65535 || n_in <= 0 || n_out <= 0 || R < 0 || rot_dims > R ||
      (rot_dims >= 0 && (rot_dims % 2 || out_head_stride < n_out + R || !positions ||
                         (rot_dims > 0 && (!cos_t || !sin_t)))))
    return EK_ERR_ARG;
  if (w == nullptr)
    return rot_dims < 0 ? 0
                        : (int)launch_pdl(head_tail_kernel<T>, dim3(n_tokens), dim3(256), 0, stream, out, out_row_stride,
                                          out_head_stride, in, in_row_stride, in_head_stride, heads, n_in, n_out, R, rot_dims,
                                          cos_t, sin_t, positions);
  if constexpr (std::is_same_v<T, bf16>) {
    // whole steps of 16 inputs, 16-byte pieces of weights and inputs, and what they take of shared memory without asking
    const bool by_mma = n_in % 16 == 0 && n_out % 8 == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)in & 15) == 0 &&
                        in_row_stride % 8 == 0 && in_head_stride % 8 == 0 && head_mma_smem(n_in) <= 40 * 1024;
    if (by_mma) {
      const dim3 grid((n_tokens + kHeadTokens - 1) / kHeadTokens, heads,
                      (n_out + kHeadOuts - 1) / kHeadOuts + (rot_dims >= 0 ? 1 : 0));
      if (grid.z > 65535) return EK_ERR_ARG;
      return (int)launch_pdl(head_linear_mma_kernel, grid, dim3(kHeadThreads), head_mma_smem(n_in), stream, out, out_row_stride,
                             out_head_stride, in, in_row_stride, in_head_stride, w, n_tokens, n_in, n_out, R, rot_dims, cos_t,
                             sin_t, positions);
    }
  }
  const int width = n_in + (rot_dims >= 0 ? R : 0);
  const size_t smem = (size_t)kHeadTokens * width * sizeof(float);
  if (smem > 200 * 1024) return EK_ERR_ARG;
  if (smem > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(head_linear_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid((n_tokens + kHeadTokens - 1) / kHeadTokens, heads, (n_out + kHeadOuts - 1) / kHeadOuts);
  if (grid.z > 65535) return EK_ERR_ARG;
  return (int)launch_pdl(head_linear_kernel<T>, grid, dim3(kHeadThreads), smem, stream, out, out_row_stride, out_head_stride, in, in_row_stride,
                         in_head_stride, w, n_tokens, n_in, n_out, R, rot_dims, cos_t, sin_t, positions);
}

}  // namespace ek

#define EK_INSTANTIATE(SUFFIX, T)                                                                     \
  EK_EXPORT int ek_latent_prepare_##SUFFIX(                                                           \
      void* cq, const float* proj, int proj_stride, const float* gain_q, const float* gain_kv,        \
      float eps, const float* cos_t, const float* sin_t, int rot_dims, const int* positions,          \
      const int* token_slot, void* pages, const int* block_table, int table_stride, int n_tokens,     \
      int QR, int C, int R, int D, int write_cache, cudaStream_t stream) {                            \
    using namespace ek;                                                                               \
    if (n_tokens <= 0) return 0;                                                                      \
    if (QR < 0 || (QR == 0 && gain_q) || (QR > 0 && !cq) || C <= 0 || R < 0 || D < C + R ||           \
        rot_dims < 0 || rot_dims > R || rot_dims % 2 || proj_stride < QR + C + R)                     \
      return EK_ERR_ARG;                                                                              \
    return (int)launch_pdl(latent_prepare_kernel<T>, dim3(n_tokens), dim3(QR > 2048 ? 512 : 256), 0, stream, (T*)cq, \
                           proj, proj_stride, gain_q, gain_kv, eps, cos_t, sin_t, rot_dims, positions,  \
                           token_slot, (T*)pages, block_table, table_stride, QR, C, R, D, write_cache); \
  }                                                                                                   \
  EK_EXPORT int ek_head_linear_##SUFFIX(                                                              \
      void* out, int out_row_stride, int out_head_stride, const void* in, int in_row_stride,          \
      int in_head_stride, const void* w, int n_tokens, int heads, int n_in, int n_out, int R,         \
      int rot_dims, const float* cos_t, const float* sin_t, const int* positions,                     \
      cudaStream_t stream) {                                                                          \
    return ek::launch_head_linear<T>((T*)out, out_row_stride, out_head_stride, (const T*)in,          \
                                     in_row_stride, in_head_stride, (const T*)w, n_tokens, heads,     \
                                     n_in, n_out, R, rot_dims, cos_t, sin_t, positions, stream);      \
  }

EK_INSTANTIATE(f32, float)
EK_INSTANTIATE(bf16, ek::bf16)
