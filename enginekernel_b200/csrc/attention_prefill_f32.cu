// Attention of prompts in true 32-bit: several new tokens per sequence against the paged cache, on the
// CUDA cores.  Same formula and options as the general kernel (attention_generic.cu), which computes one
// token and head a block and reads every key and value row for each of them from L2; here a block takes 64
// consecutive tokens of one sequence and one query head, and every key page serves all of them.
//
// Bound by the FMA pipes and the shared-memory reads that feed them (as the 32-bit product,
// gemm_f32.cu).  128 threads: 8 rows x 4 keys a thread for the scores, the same 8 rows x a sixteenth of
// the head a thread for the weighted sum of values, so that a row's maximum and sum stay with the 16
// lanes that hold its scores and its result.  Keys and values of a page take turns in one buffer (the
// values are on their way while the softmax runs): two blocks fit an SM, and one computes while the
// other waits.  Pages are aligned to the sequence, so what a token adds up, and in which order, does
// not depend on which other tokens share its block.
#include "common.cuh"

namespace ek {

constexpr int kF32Rows = 64, kF32Keys = EK_PAGE, kF32Threads = 128;
constexpr int kF32PLd = kF32Keys + 4;
__host__ __device__ constexpr size_t f32_attn_smem(int dmax) {      // Q, K or V, P
  return (size_t)(kF32Rows * (dmax + 4) + kF32Keys * (dmax + 4) + kF32Rows * kF32PLd) * 4;
}

// grid (query heads, tiles upper bound).  Head sizes up to DMAX, multiples of 4; padded with zeros.
template <int DMAX>
__global__ void __launch_bounds__(kF32Threads)
attention_prefill_f32_kernel(float* __restrict__ out, const float* __restrict__ q, int q_row_stride,
                             const int* __restrict__ positions, const int* __restrict__ token_slot,
                             const int* __restrict__ cu_seqlens, int n_seqs, PagedKV cache, int n_q_heads,
                             float scale, int window, float sink, const float* __restrict__ sinks, int keep_first,
                             const float* __restrict__ gate, int gate_stride, int chunk, float softcap) {
  constexpr int LD = DMAX + 4;
  constexpr int GROUPS = DMAX / 64;                // groups of 4 neighbouring dimensions a thread
  extern __shared__ __align__(16) float f32_smem[];
  float* q_s = f32_smem;                           // [64][LD]
  float* kv_s = q_s + kF32Rows * LD;               // [64][LD]
  float* p_s = kv_s + kF32Keys * LD;               // [64][kF32PLd]
  __shared__ int tile_info[3];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;     // rows ty + 8 i, keys tx + 16 j
  const int h = blockIdx.x, D = cache.head_dim;
  const int kv_head = h / (n_q_heads / cache.heads);

  if (tid == 0) {
    int idx = blockIdx.y, found = -1, first = 0, count = 0;
    for (int b = 0; b < n_seqs; ++b) {
      const int n = cu_seqlens[b + 1] - cu_seqlens[b];
      const int tiles = (n + kF32Rows - 1) / kF32Rows;
      if (idx < tiles) {
        const int tile = tiles - 1 - idx;          // long key ranges first
        found = b;
        first = cu_seqlens[b] + tile * kF32Rows;
        count = min(kF32Rows, n - tile * kF32Rows);
        break;
      }
      idx -= tiles;
    }
    tile_info[0] = first; tile_info[1] = count; tile_info[2] = found;
  }
  __syncthreads();
  if (tile_info[2] < 0) return;
  const int t0 = tile_info[0], n_rows = tile_info[1];
  const int pos0 = positions[t0];
  if (pos0 < 0) {                                  // rows of a finished sequence: zeros
    for (int i = tid; i < n_rows * D; i += kF32Threads)
      out[((size_t)(t0 + i / D) * n_q_heads + h) * D + i % D] = 0.f;
    return;
  }
  const int* table = cache.block_table + (size_t)token_slot[t0] * cache.table_stride;
  const int page_lo = first_key(pos0, window, chunk) / kF32Keys, page_hi = (pos0 + n_rows - 1) / kF32Keys;
  const int n_first = keep_first > 0 ? min((keep_first + kF32Keys - 1) / kF32Keys, page_lo) : 0;
  const int n_pages = n_first + page_hi - page_lo + 1;

  // rows of DMAX values: the head's (16 bytes a copy), zeros behind them and below the last row
  auto copy_rows = [&](float* dst, const float* src, size_t stride, int rows) {
    constexpr int PIECES = DMAX / 4;
#pragma unroll 4
    for (int i = tid; i < 64 * PIECES; i += kF32Threads) {
      const int r = i / PIECES, c = i % PIECES * 4;
      const int bytes = r < rows && c < D ? 16 : 0;
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + r * LD + c);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(bytes ? src + r * stride + c : src),
                   "r"(bytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto landed = [&] {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  };
  auto page_of = [&](int i) { return i < n_first ? i : page_lo + (i - n_first); };
  auto page_rows = [&](int p) { return min(kF32Keys, pos0 + n_rows - p * kF32Keys); };   // keys that are there
  auto page_at = [&](const void* base, int p) {
    return (const float*)base + ((size_t)table[p] * cache.heads + kv_head) * kF32Keys * (size_t)D;
  };

  copy_rows(q_s, q + (size_t)t0 * q_row_stride + (size_t)h * D, q_row_stride, n_rows);
  copy_rows(kv_s, page_at(cache.k, page_of(0)), D, page_rows(page_of(0)));

  float o[8][4 * GROUPS], m[8], l[8];
  int first[8];                                    // the first key of the window that row i sees
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
    first[i] = first_key(pos0 + ty + 8 * i, window, chunk);
#pragma unroll
    for (int c = 0; c < 4 * GROUPS; ++c) o[i][c] = 0.f;
  }
  landed();
  for (int i = tid; i < kF32Rows * DMAX; i += kF32Threads) q_s[i / DMAX * LD + i % DMAX] *= scale;
  __syncthreads();

  for (int it = 0; it < n_pages; ++it) {
    const int page = page_of(it), key0 = page * kF32Keys;
    if (it > 0) landed();                          // the page's keys
    float s[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < DMAX; d += 4) {
      float4 kv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(kv_s + (tx + 16 * j) * LD + d);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(q_s + (ty + 8 * i) * LD + d);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[i][j] = fmaf(a.w, kv[j].w, fmaf(a.z, kv[j].z, fmaf(a.y, kv[j].y, fmaf(a.x, kv[j].x, s[i][j]))));
      }
    }
    __syncthreads();                               // the keys have been read
    copy_rows(kv_s, page_at(cache.v, page), D, page_rows(page));

    // softmax: scores of a row are with 16 lanes of a warp
    const bool edge = key0 + kF32Keys - 1 > pos0 || key0 < first_key(pos0 + n_rows - 1, window, chunk);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int p = pos0 + ty + 8 * i;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v = s[i][j];
        if (softcap > 0.f) v = softcap * tanhf(v / softcap);
        const int key = key0 + tx + 16 * j;
        if (edge && (key > p || (key < first[i] && key >= keep_first))) v = -INFINITY;
        s[i][j] = v;
        mx = fmaxf(mx, v);
      }
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float m_new = fmaxf(m[i], mx);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;       // (no key of this row so far)
      const float alpha = expf(m[i] - m_use);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = expf(s[i][j] - m_use);
        sum += e;
        p_s[(ty + 8 * i) * kF32PLd + tx + 16 * j] = e;
      }
      m[i] = m_new;
      l[i] = l[i] * alpha + sum;                   // (this lane's keys; summed over the lanes at the end)
#pragma unroll
      for (int c = 0; c < 4 * GROUPS; ++c) o[i][c] *= alpha;
    }
    landed();                                      // the page's values, and everyone's weights
    // A weight of 0 takes nothing from a key that a row does not see, unless that key's value is infinite or
    // not a number: pages on an edge look for such values and then leave those terms out one by one.
    int strange = 0;
    if (edge)
      for (int i = tid; i < kF32Keys * DMAX; i += kF32Threads)
        strange |= !(fabsf(kv_s[i / DMAX * LD + i % DMAX]) <= 3.402823466e38f);
    if (edge && __syncthreads_or(strange)) {
      for (int key = 0; key < kF32Keys; ++key)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float w = p_s[(ty + 8 * i) * kF32PLd + key];
#pragma unroll
          for (int c = 0; c < 4 * GROUPS; ++c)
            if (w != 0.f) o[i][c] = fmaf(w, kv_s[key * LD + c / 4 * 64 + tx * 4 + c % 4], o[i][c]);
        }
    } else {
#pragma unroll 2
      for (int key = 0; key < kF32Keys; key += 4) {
        float4 v[4][GROUPS];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
          for (int g = 0; g < GROUPS; ++g)
            v[kk][g] = *reinterpret_cast<const float4*>(kv_s + (key + kk) * LD + g * 64 + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 w4 = *reinterpret_cast<const float4*>(p_s + (ty + 8 * i) * kF32PLd + key);
          const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
              o[i][4 * g] = fmaf(w[kk], v[kk][g].x, o[i][4 * g]);
              o[i][4 * g + 1] = fmaf(w[kk], v[kk][g].y, o[i][4 * g + 1]);
              o[i][4 * g + 2] = fmaf(w[kk], v[kk][g].z, o[i][4 * g + 2]);
              o[i][4 * g + 3] = fmaf(w[kk], v[kk][g].w, o[i][4 * g + 3]);
            }
        }
      }
    }
    __syncthreads();                               // values and weights have been read
    if (it + 1 < n_pages) {
      const int next = page_of(it + 1);
      copy_rows(kv_s, page_at(cache.k, next), D, page_rows(next));
    }
  }

  if (sinks != nullptr) sink = sinks[h];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int x = 8; x > 0; x >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);
    const int r = ty + 8 * i;
    if (r >= n_rows) continue;
    if (sink > -INFINITY && l[i] > 0.f) l[i] += expf(sink - m[i]);
    float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    if (gate != nullptr) inv *= 1.f / (1.f + expf(-gate[(size_t)(t0 + r) * gate_stride + h]));
    float* to = out + ((size_t)(t0 + r) * n_q_heads + h) * D;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      const int c = g * 64 + tx * 4;
      if (c < D)
        *reinterpret_cast<float4*>(to + c) =
            make_float4(o[i][4 * g] * inv, o[i][4 * g + 1] * inv, o[i][4 * g + 2] * inv, o[i][4 * g + 3] * inv);
    }
  }
}

}  // namespace ek

// Several new tokens per sequence, 32-bit: sequence b owns rows cu_seqlens[b] .. cu_seqlens[b + 1] of q, which
// stand at consecutive positions; keys and values are in the pages.  Head sizes up to 128, multiples of 4, every
// operand on 16-byte boundaries.
EK_EXPORT int ek_attention_prefill_f32(float* out, const float* q, int q_row_stride, const int* positions,
                                       const int* token_slot, const int* cu_seqlens, int n_seqs, int n_tokens,
                                       const float* k_pages, const float* v_pages, const int* block_table,
                                       int table_stride, int n_q_heads, int n_kv_heads, int head_dim, float scale,
                                       int window, float sink, const float* sinks, int keep_first, const float* gate,
                                       int gate_stride, int chunk, float softcap, cudaStream_t stream) {
  using namespace ek;
  if (n_tokens <= 0 || n_seqs <= 0) return 0;
  const long long tiles = (long long)(n_tokens / kF32Rows) + n_seqs;
  if (chunk < 0 || (chunk > 0 && (window > 0 || keep_first > 0)) || head_dim <= 0 || head_dim > 128 || head_dim % 4 ||
      n_kv_heads <= 0 || n_q_heads % n_kv_heads || q_row_stride % 4 || tiles > 65535 ||
      (((uintptr_t)out | (uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15))
    return EK_ERR_ARG;
  const PagedKV cache{(void*)k_pages, (void*)v_pages, block_table, table_stride, n_kv_heads, head_dim};
  auto kernel = head_dim <= 64 ? attention_prefill_f32_kernel<64> : attention_prefill_f32_kernel<128>;
  const size_t smem = f32_attn_smem(head_dim <= 64 ? 64 : 128);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  kernel<<<dim3(n_q_heads, (unsigned)tiles), kF32Threads, smem, stream>>>(
      out, q, q_row_stride, positions, token_slot, cu_seqlens, n_seqs, cache, n_q_heads, scale, window, sink, sinks,
      window > 0 ? keep_first : 0, gate, gate_stride, chunk, softcap);
  EK_RETURN_LAUNCH_STATUS();
}
