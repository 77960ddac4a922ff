// Routed experts: a router that picks `top` of E small feed-forwards per token, and the experts'
// products for the tokens that chose them.
//
//   route     scores = softmax(logits) over all experts (32-bit); experts form `n_groups` equal
//             groups of neighbours, a group's score is its best expert's, only experts of the
//             `keep` best groups can be chosen; the `top` largest of those; weights = chosen
//             scores / (their sum + 1e-20) * scale.  A warp a token.  `among_chosen`: the weights are
//             the softmax over the chosen logits alone (times scale), taken from the logits with the
//             chosen maximum off, so that no score can vanish against an unchosen expert's.  `mode` 2: scores
//             are sigmoids of the logits, each for itself; the weights are the chosen scores times scale,
//             not divided by their sum.  `mode` 3: softmax scores over all experts as weights (times scale, not
//             divided by their sum); `correction` [E] (any sign) joins the scores for the choice only.
//             Numbers from the plan's E on name experts without weights whose output is the input itself:
//             the plan leaves their pairs out and `combine` adds weight * input.
//   plan      the (token, choice) pairs sorted by expert, and the row tiles of every expert's
//             stretch, made on the device: the host never sees who chose what.
//   expert product  out[row] = f(x[row] . W_e^T) over the tiles of the plan: FFMA with 32-bit
//             sums in ascending k (the 32-bit path, and 16-bit rows that cannot be read 16 bytes
//             at a time; the others run on pairs of SMs, moe_pair.cu); either way a
//             pair's result does not depend on its neighbours.  The up form gathers its rows by
//             token and applies the activation, the down form scales by the pair's weight and
//             scatters 32-bit rows by pair.  `gated` up form: the expert's weight rows alternate
//             gate, up, gate, up ...; column pair (2c, 2c + 1) of the product gives out[c] =
//             act(gate) * up from the 32-bit sums (N counts the weight rows, the output has N / 2).
//             `row_weight` (up form): a pair's weight multiplies its row of the product before the activation,
//             which is the product of the weighted input; `limit` belongs to the clamped activation.
//   combine   out[t] = sum over the token's choices, in the order they were chosen (a choice that names an
//             expert without weights adds weight * x[t]) (+ add[t], the result of an expert that every token shares).
#include "moe_common.cuh"

namespace ek {

__device__ __forceinline__ void warp_argmax(float& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
  }
}

constexpr int kRouteWarps = 4;

// logits [T, >= E] 32-bit (rows row_stride apart) -> sel_expert [T, top] int32, sel_weight [T, top] 32-bit.
__global__ void __launch_bounds__(kRouteWarps * 32)
moe_route_kernel(int* __restrict__ sel_expert, float* __restrict__ sel_weight,
                 const float* __restrict__ logits, int row_stride, int n_tokens, int E, int n_groups, int keep, int top,
                 float scale, int mode, const float* __restrict__ correction) {
  // mode 0: softmax scores, divided by the chosen ones' sum; 1: softmax over the chosen; 2: sigmoids as they are;
  // 3: softmax scores as they are, chosen by score + correction
  const bool among_chosen = mode == 1 || mode == 2;     // (candidates are compared by their logits)
  extern __shared__ float route_s[];            // per warp: scores [E], candidates [E], groups [n_groups]
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * kRouteWarps + warp;
  if (t >= n_tokens) return;
  float* s = route_s + (size_t)warp * (2 * E + n_groups);
  float* cand = s + E;
  float* gs = cand + E;
  const float* z = logits + (size_t)t * row_stride;
  float m = -INFINITY;
  for (int e = lane; e < E; e += 32) m = fmaxf(m, z[e]);
  m = warp_max(m);
  float sum = 0.f;
  for (int e = lane; e < E; e += 32) { const float x = expf(z[e] - m); s[e] = x; sum += x; }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
  // candidates: the scores; with weights among the chosen the logits themselves, so that the order of
  // two experts whose scores both round to nothing is still the order of their logits
  const float shut = mode != 0 ? -INFINITY : -2.f;
  for (int e = lane; e < E; e += 32) {
    s[e] *= inv;
    cand[e] = among_chosen ? z[e] : correction != nullptr ? s[e] + correction[e] : s[e];
  }
  __syncwarp();
  if (n_groups > 1 && keep < n_groups) {
    const int per = E / n_groups;
    for (int g = lane; g < n_groups; g += 32) {
      float best = -1.f;
      for (int e = g * per; e < (g + 1) * per; ++e) best = fmaxf(best, s[e]);
      gs[g] = best;
    }
    __syncwarp();
    for (int round = 0; round < keep; ++round) {
      float bv = -2.f; int bi = 0x7fffffff;
      for (int g = lane; g < n_groups; g += 32)
        if (gs[g] > bv) { bv = gs[g]; bi = g; }
      warp_argmax(bv, bi);
      if (lane == 0) gs[bi] = -3.f;             // kept
      __syncwarp();
    }
    for (int e = lane; e < E; e += 32)
      if (gs[e / per] != -3.f) cand[e] = among_chosen ? -INFINITY : -1.f;
    __syncwarp();
  }
  float total = 0.f;
  for (int k = 0; k < top; ++k) {
    float bv = shut; int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32)
      if (cand[e] > bv) { bv = cand[e]; bi = e; }
    warp_argmax(bv, bi);
    if (bi >= E) bi = 0;                        // (no finite candidate left: logits that are not numbers)
    const float sc = s[bi];
    total += sc;
    if (lane == 0) {
      sel_expert[(size_t)t * top + k] = bi;
      sel_weight[(size_t)t * top + k] = sc;     // scaled below
      cand[bi] = shut;
    }
    __syncwarp();
  }
  if (mode == 2) {
    __syncwarp();
    for (int k = lane; k < top; k += 32) {
      const float x = z[sel_expert[(size_t)t * top + k]];
      sel_weight[(size_t)t * top + k] = scale / (1.f + expf(-x));
    }
    return;
  }
  if (among_chosen) {                           // softmax over the chosen logits: the first chosen is the largest
    __syncwarp();
    const float z0 = z[sel_expert[(size_t)t * top]];
    float den = 0.f;
    for (int k = 0; k < top; ++k) den += expf(z[sel_expert[(size_t)t * top + k]] - z0);
    for (int k = lane; k < top; k += 32)
      sel_weight[(size_t)t * top + k] = expf(z[sel_expert[(size_t)t * top + k]] - z0) / den * scale;
    return;
  }
  const float f = mode == 3 ? scale : scale / (total + 1e-20f);
  for (int k = lane; k < top; k += 32) sel_weight[(size_t)t * top + k] *= f;
}

constexpr int kTileRows = 64;

// One block.  sel_expert [P] -> sorted_pair [P] (pairs grouped by expert), tiles [max_tiles][3] =
// (expert, first sorted row, rows), n_tiles[0].  Tiles hold up to `tile_rows` rows; with `even` > 0 an expert's
// tiles are as few as that allows and equal, up to the next multiple of `even` rows.
__global__ void __launch_bounds__(1024)
moe_plan_kernel(int* __restrict__ sorted_pair, int* __restrict__ tiles, int* __restrict__ n_tiles,
                const int* __restrict__ sel_expert, int P, int E, int tile_rows, int even) {
  extern __shared__ int plan_s[];               // counts [E], first row [E], first tile [E + 1]
  auto rows_of = [&](int n) {                   // rows of the tiles of an expert with n pairs
    if (even <= 0 || n <= 0) return tile_rows;
    const int tiles_n = (n + tile_rows - 1) / tile_rows, each = (n + tiles_n - 1) / tiles_n;
    return (each + even - 1) / even * even;
  };
  pdl_launch_dependents();
  pdl_wait();
  int* counts = plan_s;
  int* first = counts + E;
  int* tile0 = first + E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) counts[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int e = sel_expert[p];
    if (e >= 0 && e < E) atomicAdd(&counts[e], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {                       // first rows and first tiles: a scan, a lane an expert
    const int lane = threadIdx.x;
    int row = 0, tile = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, n = e < E ? counts[e] : 0, each = rows_of(n), t = (n + each - 1) / each;
      int rows_to = n, tiles_to = t;            // up to and with this lane's
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int r = __shfl_up_sync(0xffffffffu, rows_to, o), q = __shfl_up_sync(0xffffffffu, tiles_to, o);
        if (lane >= o) { rows_to += r; tiles_to += q; }
      }
      if (e < E) {
        first[e] = row + rows_to - n;
        tile0[e] = tile + tiles_to - t;
      }
      row += __shfl_sync(0xffffffffu, rows_to, 31);
      tile += __shfl_sync(0xffffffffu, tiles_to, 31);
    }
    if (lane == 0) {
      tile0[E] = tile;
      n_tiles[0] = tile;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int n = counts[e], each = rows_of(n);
    for (int i = 0, tile = tile0[e]; i < n; i += each, ++tile) {
      tiles[3 * tile] = e;
      tiles[3 * tile + 1] = first[e] + i;
      tiles[3 * tile + 2] = min(each, n - i);
    }
    counts[e] = first[e];                       // from here on: the next free row of the expert
  }
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int e = sel_expert[p];
    if (e >= 0 && e < E) sorted_pair[atomicAdd(&counts[e], 1)] = p;
  }
}

// grid (max tiles, column tiles).  UP: a[row] = x[pair / top], out T [sorted row][N] = act(.).
// DOWN: a[row] = in[sorted row], out 32-bit [pair][N] = weight[pair] * (.).
template <typename T, bool UP>
__global__ void __launch_bounds__(256)
moe_expert_product_kernel(void* __restrict__ out_, const T* __restrict__ a, const T* __restrict__ w,
                          const int* __restrict__ tiles, const int* __restrict__ n_tiles,
                          const int* __restrict__ sorted_pair, const float* __restrict__ pair_weight,
                          int top, int N, int K, int act, int gated, float limit) {
  constexpr int BM = kTileRows, BN = 64, BK = 16, TM = 4, TN = 4, PAD = 4;
  __shared__ __align__(16) float As[BK][BM + PAD];
  __shared__ __align__(16) float Ws[BK][BN + PAD];
  __shared__ int src_row[BM];
  __shared__ int pair_s[BM];
  pdl_launch_dependents();
  pdl_wait();
  if ((int)blockIdx.x >= n_tiles[0]) return;
  const int e = tiles[3 * blockIdx.x], row0 = tiles[3 * blockIdx.x + 1], rows = tiles[3 * blockIdx.x + 2];
  const int tid = threadIdx.x;
  if (tid < BM) {
    const int p = tid < rows ? sorted_pair[row0 + tid] : -1;
    pair_s[tid] = p;
    src_row[tid] = p < 0 ? -1 : (UP ? p / top : row0 + tid);
  }
  __syncthreads();
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int n0 = blockIdx.y * BN;
  const T* we = w + (size_t)e * N * K;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int idx = tid; idx < BM * BK; idx += 256) {
      const int row = idx / BK, kk = idx % BK;
      const int src = src_row[row], gk = k0 + kk;
      As[kk][row] = (src >= 0 && gk < K) ? to_f<T>(a[(size_t)src * K + gk]) : 0.f;
    }
    for (int idx = tid; idx < BN * BK; idx += 256) {
      const int row = idx / BK, kk = idx % BK;
      const int gn = n0 + row, gk = k0 + kk;
      Ws[kk][row] = (gn < N && gk < K) ? to_f<T>(we[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float av[TM], bv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = ty * TM + i;
    if (r >= rows) continue;
    const float rw = UP && pair_weight != nullptr ? pair_weight[pair_s[r]] : 1.f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= N) continue;
      if (UP && gated) {                          // columns (gn, gn + 1) = (gate, up); N is even
        if (!(j & 1)) ((T*)out_)[(size_t)(row0 + r) * (N / 2) + gn / 2] =
            from_f<T>(gated_value(acc[i][j] * rw, acc[i][j + 1] * rw, act, limit));
      } else if (UP) {
        ((T*)out_)[(size_t)(row0 + r) * N + gn] = from_f<T>(activate(acc[i][j] * rw, act));
      } else {
        const int p = pair_s[r];
        ((float*)out_)[(size_t)p * N + gn] = acc[i][j] * (pair_weight != nullptr ? pair_weight[p] : 1.f);
      }
    }
  }
}

// out[sorted row] = x[token of the pair], 16 bytes a thread: the rows of the up product side by side.  A warp a row.
__global__ void __launch_bounds__(256)
moe_gather_kernel(uint4* __restrict__ out, const uint4* __restrict__ x, const int* __restrict__ sorted_pair,
                  const int* __restrict__ tiles, const int* __restrict__ n_tiles, int P, int top, int pieces) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int last = n_tiles[0] - 1;               // (pairs whose expert has no weights have no row)
  if (last < 0 || row >= min(P, tiles[3 * last + 1] + tiles[3 * last + 2])) return;
  const uint4* from = x + (size_t)(sorted_pair[row] / top) * pieces;
  uint4* to = out + (size_t)row * pieces;
#pragma unroll 8
  for (int i = lane; i < pieces; i += 32) to[i] = from[i];
}

// out[t, :] = sum_k pair_out[t * top + k, :], k ascending (+ add[t, :]).  A choice k whose expert number is E or more
// (`chosen` given) has no row in pair_out: weight[t, k] * x[t, :] takes its place.  Four values a thread when `vec`.
template <typename T>
__global__ void __launch_bounds__(256)
moe_combine_kernel(T* __restrict__ out, const float* __restrict__ pair_out, int top, int width,
                   const T* __restrict__ add, const int* __restrict__ chosen, const float* __restrict__ weight,
                   const T* __restrict__ x, int E, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t t = blockIdx.x;
  if (vec) {                                     // (top <= 32: which choices are the input itself, one bit each)
    unsigned own = 0;
    if (chosen)
      for (int k = 0; k < top; ++k) own |= (chosen[t * top + k] >= E ? 1u : 0u) << k;
    for (int i = threadIdx.x * 4; i < width; i += blockDim.x * 4) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xv = own ? Vec4<T>::load(x + t * width + i) : a;
#pragma unroll 4
      for (int k = 0; k < top; ++k) {
        const bool mine = own >> k & 1u;
        float4 v = xv;
        if (!mine) v = *reinterpret_cast<const float4*>(pair_out + (t * top + k) * width + i);
        const float w = mine ? weight[t * top + k] : 1.f;
        a.x = fmaf(w, v.x, a.x); a.y = fmaf(w, v.y, a.y); a.z = fmaf(w, v.z, a.z); a.w = fmaf(w, v.w, a.w);
      }
      if (add) {
        const float4 s = Vec4<T>::load(add + t * width + i);
        a.x += s.x; a.y += s.y; a.z += s.z; a.w += s.w;
      }
      Vec4<T>::store(out + t * width + i, a);
    }
    return;
  }
  for (int i = threadIdx.x; i < width; i += blockDim.x) {
    float a = 0.f;
    for (int k = 0; k < top; ++k)
      a += chosen && chosen[t * top + k] >= E ? weight[t * top + k] * to_f<T>(x[t * width + i])
                                              : pair_out[(t * top + k) * width + i];
    if (add) a += to_f<T>(add[t * width + i]);
    out[t * width + i] = from_f<T>(a);
  }
}

}  // namespace ek

EK_EXPORT int ek_moe_tile_rows() { return ek::kTileRows; }

EK_EXPORT int ek_moe_route(int* sel_expert, float* sel_weight, const float* logits, int row_stride, int n_tokens, int E,
                           int n_groups, int keep, int top, float scale, int mode,
                           const float* correction, cudaStream_t stream) {
  using namespace ek;
  if (n_tokens <= 0) return 0;
  if (E <= 0 || row_stride < E || top <= 0 || top > E || n_groups < 1 || E % n_groups || keep < 1 || keep > n_groups ||
      top > keep * (E / n_groups) || mode < 0 || mode > 3 || (mode >= 2 && keep < n_groups) ||
      (correction && mode != 3))
    return EK_ERR_ARG;
  const size_t smem = (size_t)kRouteWarps * (2 * E + n_groups) * sizeof(float);
  if (smem > 200 * 1024) return EK_ERR_ARG;
  if (smem > 40 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(moe_route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  moe_route_kernel<<<(n_tokens + kRouteWarps - 1) / kRouteWarps, kRouteWarps * 32, smem, stream>>>(
      sel_expert, sel_weight, logits, row_stride, n_tokens, E, n_groups, keep, top, scale, mode, correction);
  EK_RETURN_LAUNCH_STATUS();
}

EK_EXPORT int ek_moe_plan(int* sorted_pair, int* tiles, int* n_tiles, const int* sel_expert, int P, int E,
                          int tile_rows, int even, cudaStream_t stream) {
  if (P <= 0) return 0;
  if (E <= 0 || E > 8192 || tile_rows <= 0 || even < 0 || (even > 0 && tile_rows % even)) return EK_ERR_ARG;
  ek::moe_plan_kernel<<<1, 1024, (size_t)(3 * E + 1) * sizeof(int), stream>>>(sorted_pair, tiles, n_tiles,
                                                                             sel_expert, P, E, tile_rows, even);
  EK_RETURN_LAUNCH_STATUS();
}

// out [P, width] = x [T, width] by the plan's order; bfloat16 rows of whole 16-byte pieces.
EK_EXPORT int ek_moe_gather(void* out, const void* x, const int* sorted_pair, const int* tiles, const int* n_tiles,
                            int P, int top, int width, cudaStream_t stream) {
  if (P <= 0) return 0;
  if (top <= 0 || width <= 0 || width % 8 || ((uintptr_t)x & 15) || ((uintptr_t)out & 15)) return EK_ERR_ARG;
  return (int)ek::launch_pdl(ek::moe_gather_kernel, dim3((P + 7) / 8), dim3(256), 0, stream, (uint4*)out,
                             (const uint4*)x, sorted_pair, tiles, n_tiles, P, top, width / 8);
}

#define EK_INSTANTIATE(SUFFIX, T)                                                                     \
  EK_EXPORT int ek_moe_expert_up_##SUFFIX(void* out, const void* x, const void* w, const int* tiles,  \
                                          const int* n_tiles, const int* sorted_pair, int max_tiles,  \
                                          int top, int N, int K, int act, int gated, float limit,     \
                                          const float* row_weight, cudaStream_t stream) {             \
    using namespace ek;                                                                               \
    if (max_tiles <= 0) return 0;                                                                     \
    if (N <= 0 || K <= 0 || top <= 0 || (N + 63) / 64 > 65535 || (gated && N % 2) ||         \
        (act == ACT_CLAMPED && !(gated && limit > 0.f)))                                              \
      return EK_ERR_ARG;                                                                              \
    dim3 grid(max_tiles, (N + 63) / 64);                                                              \
    moe_expert_product_kernel<T, true><<<grid, 256, 0, stream>>>(                                     \
        out, (const T*)x, (const T*)w, tiles, n_tiles, sorted_pair, row_weight, top, N, K, act, gated, limit); \
    EK_RETURN_LAUNCH_STATUS();                                                                        \
  }                                                                                                   \
  EK_EXPORT int ek_moe_expert_down_##SUFFIX(float* out, const void* a, const void* w, const int* tiles, \
                                            const int* n_tiles, const int* sorted_pair,               \
                                            const float* pair_weight, int max_tiles, int N, int K,    \
                                            cudaStream_t stream) {                                    \
    using namespace ek;                                                                               \
    if (max_tiles <= 0) return 0;                                                                     \
    if (N <= 0 || K <= 0 || (N + 63) / 64 > 65535) return EK_ERR_ARG;                                 \
    dim3 grid(max_tiles, (N + 63) / 64);                                                              \
    moe_expert_product_kernel<T, false><<<grid, 256, 0, stream>>>(                                    \
        out, (const T*)a, (const T*)w, tiles, n_tiles, sorted_pair, pair_weight, 1, N, K, 0, 0, 0.f); \
    EK_RETURN_LAUNCH_STATUS();                                                                        \
  }                                                                                                   \
  EK_EXPORT int ek_moe_combine_##SUFFIX(void* out, const float* pair_out, int n_tokens, int top,      \
                                        int width, const void* add, const int* chosen,                \
                                        const float* weight, const void* x, int E,                    \
                                        cudaStream_t stream) {                                        \
    if (n_tokens <= 0) return 0;                                                                      \
    if (width <= 0 || top <= 0 || (chosen && (!weight || !x))) return EK_ERR_ARG;                     \
    const uintptr_t rows = (uintptr_t)out | (uintptr_t)add | (uintptr_t)x;                            \
    const int vec = width % 4 == 0 && top <= 32 && ((uintptr_t)pair_out & 15) == 0 && (rows & (4 * sizeof(T) - 1)) == 0; \
    ek::moe_combine_kernel<T><<<n_tokens, 256, 0, stream>>>((T*)out, pair_out, top, width, (const T*)add, \
                                                            chosen, weight, (const T*)x, E, vec);     \
    EK_RETURN_LAUNCH_STATUS();                                                                        \
  }

EK_INSTANTIATE(f32, float)
EK_INSTANTIATE(bf16, ek::bf16)
