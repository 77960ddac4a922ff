// Decode attention in bfloat16 with the cache pages streamed by TMA (head sizes 64 and 128,
// up to 16 query heads a KV head; and rows of 256 values that are keys and values alike, which is
// attention through a latent, any number of query heads in blocks of 16).
//
// One new token per sequence against its paged cache; the work is reading the sequence's keys
// and values once.  A block owns (token, KV head, split): a whole number of cache pages (64 keys
// each) of that head.
//   * warp 4, one thread: the producer.  A page's K and V tiles (64 x head_dim each) come by
//     cp.async.bulk.tensor into a ring of shared-memory stages, 128-byte swizzled, each stage
//     signalled by an mbarrier.  Old pages do not depend on the kernel before this one (only
//     the newest key and value do), so their copies are issued BEFORE the programmatic-launch
//     wait: the cache stream runs while the q/k/v product and the position encoding finish.
//     (Heads of 64 and 128, whose steps open with a plain launch.)
//   * warps 0-3: each takes 16 keys of a page.  The G query heads of the group are the 16 rows
//     of mma.sync.m16n8k16 (padded), K fragments come by ldmatrix, V fragments by
//     ldmatrix.trans, softmax is online in 32-bit in units of log2, P is rounded to bfloat16
//     before P.V - the same arithmetic as the register-streaming kernel in
//     attention_decode_bf16.cu, which remains for the other head sizes.
//   * the warps merge in shared memory; the splits of one (token, KV head) are a thread-block
//     cluster.  The (head, dimension) pairs are dealt to its blocks in equal runs; a block sends
//     its partial result for a pair, with its maximum and sum, into the shared memory of the
//     block that owns the pair (st.shared::cluster, into a buffer beside the ring, since the
//     owner may still be reading pages), and after one cluster barrier every block merges what
//     it was sent, in split order, and stores its run: no partials in global memory, no second
//     kernel, and no block has to outlive another's reads.
// (Rows of 256 spread a page's work over the warps in another way, see there.)
// The reference's counterpart is its Triton split-K flash-decoding kernel and combine kernel
// (engine/ek_kernels.py:534-615, 988-1019).  Every barrier wait is bounded and reports through
// `status`; every block of a cluster reaches the cluster barrier whatever happened to it.
#include "tc_common.cuh"

namespace ek {

// Warps beside the producer's.
template <int D>
constexpr int kDtWarps = D == 256 ? 8 : 4;
template <int D>
constexpr int kDtThreads = (kDtWarps<D> + 1) * 32;
constexpr int kDtPortableSplits = 8;         // blocks of a cluster: the portable limit
constexpr int kDtMaxSplits = 16;             // and the limit with the attribute for larger ones
// floats a block can be sent by its cluster: every (head, dimension) pair once (dealt in runs of
// pairs / splits rounded up, by rows of 256 to whole fours: up to four more a split), and (max, sum) of 16 heads from 16 splits
template <int D>
constexpr int kDtRecvO = 16 * D + (D == 256 ? 4 : 1) * kDtMaxSplits;
constexpr int kDtRecvMl = kDtMaxSplits * 16 * 2;

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                        uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1,
                                              uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16_16816(float c[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                               uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// grid (splits, kv heads, tokens); cluster (splits, 1, 1) when splits > 1.  A warp takes 16 keys of every page and keeps a
// result of its own for them; the warps merge in shared memory.
template <int D, int STAGES>
__global__ void __launch_bounds__(kDtThreads<D>)
attention_decode_tma_kernel(bf16* __restrict__ out, const bf16* q, int q_row_stride,
                            const int* positions, const int* token_slot,
                            const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, const int* block_table,
                            int table_stride, int n_kv_heads, int n_q_heads, float scale_log2,
                            int window, int* status, float sink_log2, const float* __restrict__ sinks, int chunk,
                            SoftCap cap) {
  constexpr int DB = D / 64;                       // 64-wide (128-byte) blocks of the head dimension
  constexpr uint32_t kSub = EK_PAGE * 128;         // one [64 keys x 64 dims] sub-tile: 8 KB
  constexpr uint32_t kStage = 2 * DB * kSub;    // K tile + V tile
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + STAGES * kStage);        // full[STAGES], empty[STAGES]
  // after the last page the ring is dead and holds, from its start: the warps' accumulators
  // [W][16][OS] and their (max, sum) [W][16][2].
  // A row of the accumulators is OS = D + 8 floats long, so that the rows a warp stores at once
  // (one per group of four lanes) lie on different banks.
  constexpr int OS = D + 8;
  float* o_s = (float*)smem;
  constexpr int W = kDtWarps<D>, THREADS = kDtThreads<D>;
  float* ml_s = o_s + W * 16 * OS;
  static_assert((size_t)(W * 16 * (OS + 2)) * 4 <= (size_t)STAGES * kStage,
                "merge buffers must fit the ring");
  // what the other blocks of the cluster send: [split][run] results, [split][head][2] (max, sum)
  float* recv_o = (float*)(bars + 2 * STAGES);
  float* recv_ml = recv_o + kDtRecvO<D>;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  const int split = blockIdx.x, n_splits = gridDim.x;
  const int t = blockIdx.z;
  const int kv_head = blockIdx.y, group = n_q_heads / n_kv_heads;      // query heads of the KV head
  const int head0 = kv_head * group;

  pdl_launch_dependents();
  if (tid == W * 32) {
    tma_prefetch_map(&map_k);
    tma_prefetch_map(&map_v);
  }
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), W);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Read before the wait: positions, slots and block tables must have been written by work that
  // a plain (not programmatic) launch separates from this kernel.  A step's first kernel, the
  // embedding lookup, is such a launch, so the state advance of the step before is complete here, in a
  // captured graph and in eager decoding alike.  Past L1, which may hold the step before's (common.cuh).
  const int pos = load_past_l1(positions + t);
  const int slot_t = load_past_l1(token_slot + t);
  int lo = 0, hi = -1, pg_first = 0, pg_last = -1;
  if (pos >= 0) {
    lo = first_key(pos, window, chunk);
    hi = pos;
    const int pg_lo = lo / EK_PAGE, pg_hi = hi / EK_PAGE;
    const int per = (pg_hi - pg_lo + n_splits) / n_splits;     // pages a split, rounded up
    pg_first = pg_lo + split * per;
    pg_last = min(pg_hi, pg_first + per - 1);
  }
  const int n_pages = pg_last - pg_first + 1;                  // <= 0: nothing for this split
  const int new_page = pos >= 0 ? pos / EK_PAGE : -1;          // holds the key written just now

  __syncthreads();

  bool ok = true;
  float acc[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};   // rows g and g + 8

  if (warp == W) {
    // ------------------------------------------------------------------- TMA producer: one thread, for which the
    // warp's lanes fetch 32 entries of the block table at a time
    const int* table = block_table + (size_t)(pos >= 0 ? slot_t : 0) * table_stride + pg_first;
    bool waited = false;
    const uint64_t stream_policy = l2_policy_evict_first();   // a page is read once a step
    int entry = 0;
    for (int i = 0; i < n_pages; ++i) {
      if (i % 32 == 0 && i + lane < n_pages) entry = load_past_l1(table + i + lane);
      const int page = __shfl_sync(0xffffffffu, entry, i % 32);
      if (lane == 0) {
        const int s = i % STAGES;
        if (i >= STAGES) ok = mbar_wait(empty(s), ((i / STAGES) & 1) ^ 1, status, 41);
        if (pg_first + i == new_page && !waited) {   // this page was written to by the kernel before
          pdl_wait();
          waited = true;
        }
        if (ok) {
          const int row = (page * n_kv_heads + kv_head) * EK_PAGE;
          const uint32_t dst = smem_u32(smem + s * kStage);
          mbar_expect_tx(full(s), kStage);
#pragma unroll
          for (int j = 0; j < DB; ++j) {
            tma_load_2d_hint(dst + j * kSub, &map_k, 64 * j, row, full(s), stream_policy);
            tma_load_2d_hint(dst + (DB + j) * kSub, &map_v, 64 * j, row, full(s), stream_policy);
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
    }
  } else if (warp < W) {
    // ------------------------------------------------------------------- consumers
    pdl_wait();                                  // the queries come from the kernel before
    if (n_pages > 0) {
      // Q fragments of m16n8k16 for every 16-wide step of the head dimension: rows g and g + 8
      uint32_t qa[D / 16][4];
      const bf16* qrow = q + (size_t)t * q_row_stride + (size_t)head0 * D;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const int d0 = 16 * ks + 2 * tq;
        qa[ks][0] = g < group ? *reinterpret_cast<const uint32_t*>(qrow + (size_t)g * D + d0) : 0u;
        qa[ks][1] = g + 8 < group ? *reinterpret_cast<const uint32_t*>(qrow + (size_t)(g + 8) * D + d0) : 0u;
        qa[ks][2] = g < group ? *reinterpret_cast<const uint32_t*>(qrow + (size_t)g * D + d0 + 8) : 0u;
        qa[ks][3] = g + 8 < group ? *reinterpret_cast<const uint32_t*>(qrow + (size_t)(g + 8) * D + d0 + 8) : 0u;
      }
      // this lane's row and 16-byte column inside a [64 x 64] sub-tile for the two ldmatrix forms
      const int k_row = 16 * warp + (lane & 7) + 8 * (lane >> 4), k_half = (lane >> 3) & 1;
      const int v_row = 16 * warp + (lane & 7) + 8 * ((lane >> 3) & 1), v_half = lane >> 4;
      for (int i = 0; i < n_pages; ++i) {
        const int s = i % STAGES;
        ok = mbar_wait(full(s), (i / STAGES) & 1, status, 42);
        if (!ok) break;
        const int key0 = (pg_first + i) * EK_PAGE + 16 * warp;
        if (key0 <= hi && key0 + 15 >= lo) {     // else none of this warp's 16 keys is visible
          const uint32_t k_s = smem_u32(smem + s * kStage), v_s = k_s + DB * kSub;
          float sc[2][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[0][e] = sc[1][e] = 0.f;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const int chunk = 2 * ks + k_half;               // 16-byte column of the head dimension
            uint32_t b0, b1, b2, b3;
            ldsm_x4(k_s + (chunk >> 3) * kSub + k_row * 128 + (((chunk & 7) ^ (k_row & 7)) << 4), b0, b1,
                    b2, b3);
            uint32_t* a = qa[ks];
            mma_bf16_16816(sc[0], a[0], a[1], a[2], a[3], b0, b1);
            mma_bf16_16816(sc[1], a[0], a[1], a[2], a[3], b2, b3);
          }
          // sc[j][0..1]: row g, keys key0 + 8j + 2tq + {0,1}; sc[j][2..3]: row g + 8, same keys
          float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int key = key0 + 8 * j + 2 * tq + (e & 1);
              const float score = cap.c > 0.f ? capped_log2(sc[j][e], cap) : sc[j][e] * scale_log2;
              const float v = (key >= lo && key <= hi) ? score : -INFINITY;
              sc[j][e] = v;
              mx[e >> 1] = fmaxf(mx[e >> 1], v);
            }
          float alpha[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            const float m_new = fmaxf(m_run[r], mx[r]);      // finite: a key of the unit is visible
            alpha[r] = exp2f(m_run[r] - m_new);
            m_run[r] = m_new;
          }
          float psum[2] = {0.f, 0.f};
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float p = exp2f(sc[j][e] - m_run[e >> 1]);
              sc[j][e] = p;
              psum[e >> 1] += p;
            }
          l_run[0] = l_run[0] * alpha[0] + psum[0];
          l_run[1] = l_run[1] * alpha[1] + psum[1];
          const uint32_t p0 = pack2_bf16(sc[0][0], sc[0][1]), p1 = pack2_bf16(sc[0][2], sc[0][3]);
          const uint32_t p2 = pack2_bf16(sc[1][0], sc[1][1]), p3 = pack2_bf16(sc[1][2], sc[1][3]);
#pragma unroll
          for (int x = 0; x < D / 16; ++x) {
            const int chunk = 2 * x + v_half;
            uint32_t b0, b1, b2, b3;
            ldsm_x4_trans(v_s + (chunk >> 3) * kSub + v_row * 128 + (((chunk & 7) ^ (v_row & 7)) << 4), b0,
                          b1, b2, b3);
            float* a0 = acc[2 * x];
            float* a1 = acc[2 * x + 1];
            a0[0] *= alpha[0]; a0[1] *= alpha[0]; a0[2] *= alpha[1]; a0[3] *= alpha[1];
            a1[0] *= alpha[0]; a1[1] *= alpha[0]; a1[2] *= alpha[1]; a1[3] *= alpha[1];
            mma_bf16_16816(a0, p0, p1, p2, p3, b0, b1);
            mma_bf16_16816(a1, p0, p1, p2, p3, b2, b3);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty(s));
      }
    }
  }

  // ------------------------------------------------------------ the warps' results, merged
  const int failed = __syncthreads_or(ok ? 0 : 1);  // every page consumed: the ring is dead
  if (!failed && warp < W) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    }
    // acc[n][e]: row g (e < 2) or g + 8, dimension 8n + 2tq + (e & 1); only the group's rows
    // are real (the others pad the MMA's 16) and only those are stored and merged
    if (g < group) {
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        *reinterpret_cast<float2*>(o_s + ((size_t)warp * 16 + g) * OS + 8 * n + 2 * tq) =
            make_float2(acc[n][0], acc[n][1]);
      if (tq == 0) {
        ml_s[(warp * 16 + g) * 2] = m_run[0];
        ml_s[(warp * 16 + g) * 2 + 1] = l_run[0];
      }
    }
    if (g + 8 < group) {
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        *reinterpret_cast<float2*>(o_s + ((size_t)warp * 16 + g + 8) * OS + 8 * n + 2 * tq) =
            make_float2(acc[n][2], acc[n][3]);
      if (tq == 0) {
        ml_s[(warp * 16 + g + 8) * 2] = m_run[1];
        ml_s[(warp * 16 + g + 8) * 2 + 1] = l_run[1];
      }
    }
  }
  __syncthreads();
  const int pairs = group * D;
  const int run = (pairs + n_splits - 1) / n_splits;           // pairs a block of the cluster owns
  if (!failed) {
    // in warp order; a thread takes (row, dimension) pairs
    for (int idx = tid; idx < pairs; idx += THREADS) {
      const int r = idx / D, d = idx % D;
      float m = -INFINITY;
#pragma unroll
      for (int w = 0; w < W; ++w) m = fmaxf(m, ml_s[(w * 16 + r) * 2]);
      float l = 0.f, o = 0.f;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const float lw = ml_s[(w * 16 + r) * 2 + 1];
        if (lw > 0.f) {
          const float f = exp2f(ml_s[(w * 16 + r) * 2] - m);
          l += lw * f;
          o += o_s[((size_t)w * 16 + r) * OS + d] * f;
        }
      }
      if (n_splits == 1) {
        // a sink: one more term exp(sink) in the denominator, with no value (-inf: none)
        const float sk = sinks ? sinks[head0 + r] * 1.4426950408889634f : sink_log2;   // per head, if given
        if (sk > -INFINITY && l > 0.f) l += exp2f(sk - m);
        out[((size_t)t * n_q_heads + head0 + r) * D + d] = __float2bfloat16_rn(l > 0.f ? o / l : 0.f);
      } else {
        const int owner = idx / run;
        st_cluster_f32(&recv_o[split * run + (idx - owner * run)], (unsigned)owner, o);
        if (d == 0) {                            // every block needs this head's maximum and sum
          for (int sp = 0; sp < n_splits; ++sp) {
            st_cluster_f32(&recv_ml[(split * 16 + r) * 2], (unsigned)sp, m);
            st_cluster_f32(&recv_ml[(split * 16 + r) * 2 + 1], (unsigned)sp, l);
          }
        }
      }
    }
  } else {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);     // let copies in flight land
  }
  if (n_splits == 1) return;

  // ------------------------------------------------------------ the splits, merged in order
  cluster_sync();                                // (every block gets here, whatever happened to it)
  if (!failed) {
    for (int slot = tid; slot < run && split * run + slot < pairs; slot += THREADS) {
      const int idx = split * run + slot;
      const int r = idx / D;
      float m = -INFINITY;
      for (int sp = 0; sp < n_splits; ++sp) m = fmaxf(m, recv_ml[(sp * 16 + r) * 2]);
      float l = 0.f, o = 0.f;
      for (int sp = 0; sp < n_splits; ++sp) {
        const float ls = recv_ml[(sp * 16 + r) * 2 + 1];
        if (ls > 0.f) {
          const float f = exp2f(recv_ml[(sp * 16 + r) * 2] - m);
          l += ls * f;
          o += recv_o[sp * run + slot] * f;
        }
      }
      const float sk = sinks ? sinks[head0 + r] * 1.4426950408889634f : sink_log2;
      if (sk > -INFINITY && l > 0.f) l += exp2f(sk - m);      // the sink, counted once
      out[((size_t)t * n_q_heads + head0) * D + idx] = __float2bfloat16_rn(l > 0.f ? o / l : 0.f);
    }
  }
}


// Rows of 256 values that are keys and values alike (attention through a latent): a stage holds them once, and grid.y
// counts blocks of 16 query heads of a KV head.  grid (splits, blocks of heads, tokens); cluster (splits, 1, 1) when
// splits > 1.
// What bounds it is the latency of one block's pages and of what follows them, not the bytes (8 tokens behind 2,048 rows
// read 8 MB, 1.3 us); of a page's 0.75 us, 0.42 are shared memory's (32 KB come in and are read twice, for the scores and for
// P.V: 811 wavefronts a page by ncu, tensor pipes 40 % active).  So two sets of four warps take the pages in turn, one set's MMAs under the other's
// fetches, and inside a set a page is spread without reading anything twice: 16 keys of the scores a warp, then 64
// dimensions of P.V of all keys, the page's maximum and P passing through shared memory.  O lies in the set's registers
// in parts, and the queries' fragments stay in registers too; only the two sets' results are merged.  Before, each
// of the eight warps kept 16 keys and a whole O of its own, fetched the queries for every page, and the merge of eight
// took 4 us of a block's 14.  All eight warps on one page, two pages a turn, did as well up to four pages a block
// and worse behind them: they meet, fetch and multiply at the same time.
// P is two bfloat16 terms.  One, taken against the set's maximum, is further from 64 bits than one against the maximum of a
// warp's 16 keys was, where a row's largest weights stay whole: errors of one token behind 300 rows .00197 against
// .00186, 64 behind 640 .00194 against .00187; with two .00165 and .00166 (a layer 0.4 us more, 2,048 rows in one block
// 25.3 -> 26.8).  Weights by ex2.approx.ftz: exp2f but for results below 2^-126, which beside the largest, 1, are nothing.
// Us by rows behind a token of 16 heads, blocks a token; before / now: 190, 1: 8.8, 6.1; 2,048, 8: 9.5, 8.0; 2,048, 1: 29.1,
// 27.2; 8,000, 1: 97.7, 95.9 (0.75 a page); 256 tokens behind 1,000, 1: 38.3, 33.0.
template <int D, int STAGES>
__global__ void __launch_bounds__(kDtThreads<D>)
attention_decode_tma_shared_kernel(bf16* __restrict__ out, const bf16* q, int q_row_stride,
                                   const int* positions, const int* token_slot,
                                   const __grid_constant__ CUtensorMap map, const int* block_table,
                                   int table_stride, int n_kv_heads, int n_q_heads, float scale_log2,
                                   int window, int* status, float sink_log2, const float* __restrict__ sinks, int chunk,
                                   SoftCap cap, const bf16* __restrict__ gate, int gate_stride) {
  constexpr int DB = D / 64;                       // 64-wide (128-byte) blocks of the head dimension
  constexpr uint32_t kSub = EK_PAGE * 128;         // one [64 keys x 64 dims] sub-tile: 8 KB
  constexpr uint32_t kStage = DB * kSub;
  constexpr int W = kDtWarps<D>, SET = W / 2;      // two sets of warps take the pages in turn
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + STAGES * kStage);        // full[STAGES], empty[STAGES], received (and 8 bytes: what follows is 16-byte aligned)
  // what the other blocks of the cluster send: [split][run] results, [split][head][2] (max, sum)
  float* recv_o = (float*)(bars + 2 * STAGES + 2);
  float* recv_ml = recv_o + kDtRecvO<D>;
  float* max_s = recv_ml + kDtRecvMl;              // [set][16 heads][warp of the set] maxima of a page, at the end the sums
  float* row_s = max_s + W * 16;                   // [set][16 heads] the set's maximum, at the end
  unsigned char* p_s = (unsigned char*)(row_s + 2 * 16);       // [set][16 heads][64 keys] P's first terms, 16-byte pieces swizzled
  unsigned char* q_s = p_s + 2 * 16 * 128;             // [16 heads][D], 16-byte pieces swizzled; then P's second terms

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  const int split = blockIdx.x, n_splits = gridDim.x;
  const int t = blockIdx.z;
  const int heads = n_q_heads / n_kv_heads;                    // query heads of a KV head
  const int row_blocks = (heads + 15) / 16;
  const int kv_head = blockIdx.y / row_blocks, row0 = 16 * (blockIdx.y % row_blocks), group = min(16, heads - row0);
  const int head0 = kv_head * heads + row0;
  const int pairs = group * D;                     // (head, dimension) pairs of the block, dealt to the splits in whole fours
  const int run = ((pairs + n_splits - 1) / n_splits + 3) & ~3;
  const int mine = max(0, min(run, pairs - split * run));

  pdl_launch_dependents();
  if (tid == W * 32) tma_prefetch_map(&map);
  const uint32_t bar0 = smem_u32(bars), received = bar0 + 16u * STAGES;
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), SET);
    }
    mbar_init(received, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (n_splits > 1) mbar_expect_tx(received, (uint32_t)(n_splits * (mine * 4 + group * 8)));
  }
  // (that barrier exists in every block of the cluster before a store from another one reaches it: arrive here, wait
  // before the first such store)
  __syncwarp();
  if (n_splits > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  // Nothing is read ahead of the wait.  A latent layer that a program drives by itself has no plain launch between two steps,
  // and every kernel of its few-row step lets the next one start at its own top: a chain of them may reach this point while
  // the step before still writes its row to an older page.
  pdl_wait();
  const int pos = positions[t];
  const int slot_t = token_slot[t];
  int lo = 0, hi = -1, pg_first = 0, pg_last = -1;
  if (pos >= 0) {
    lo = first_key(pos, window, chunk);
    hi = pos;
    const int pg_lo = lo / EK_PAGE, pg_hi = hi / EK_PAGE;
    const int per = (pg_hi - pg_lo + n_splits) / n_splits;     // pages a split, rounded up
    pg_first = pg_lo + split * per;
    pg_last = min(pg_hi, pg_first + per - 1);
    hi = min(hi, pg_last * EK_PAGE + EK_PAGE - 1);             // (the last of this split)
  }
  const int n_pages = pg_last - pg_first + 1;                  // <= 0: nothing for this split
  __syncthreads();

  bool ok = true;
  if (warp == W) {
    // ------------------------------------------------------------------- TMA producer: one thread, for which the
    // warp's lanes fetch 32 entries of the block table at a time
    const int* table = block_table + (size_t)(pos >= 0 ? slot_t : 0) * table_stride + pg_first;
    const uint64_t stream_policy = l2_policy_evict_first();   // a page is read once a step
    int entry = 0;
    for (int i = 0; i < n_pages; ++i) {
      if (i % 32 == 0 && i + lane < n_pages) entry = table[i + lane];
      const int page = __shfl_sync(0xffffffffu, entry, i % 32);
      if (lane == 0) {
        const int s = i % STAGES;
        if (i >= STAGES) ok = mbar_wait(empty(s), ((i / STAGES) & 1) ^ 1, status, 41);
        if (ok) {
          const int row = (page * n_kv_heads + kv_head) * EK_PAGE;
          const uint32_t dst = smem_u32(smem + s * kStage);
          mbar_expect_tx(full(s), kStage);
#pragma unroll
          for (int j = 0; j < DB; ++j) tma_load_2d_hint(dst + j * kSub, &map, 64 * j, row, full(s), stream_policy);
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
    }
    // (a copy of a page nobody waits for - the block gave up - lands before the block leaves)
    if (n_splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    // ------------------------------------------------------------------- the other warps
    // A page: every warp of the set scores 16 of its keys against all heads of the block; the page's maximum and P, in
    // bfloat16, pass through shared memory; then every warp adds P.V of all 64 keys to its 64 dimensions of the set's O.
    // the sink and the gate of the row that this thread stores at the end (a thread stores a second row only where the
    // splits are few), asked for here: behind everything else they took a round trip to memory of their own
    const int my_row = n_splits > 1 ? min((split * run + 4 * tid) / D, group - 1) : 0;
    float my_sink = n_splits > 1 && sinks ? sinks[head0 + my_row] * 1.4426950408889634f : sink_log2, my_gate = 1.f;
    if (n_splits > 1 && gate != nullptr) my_gate = __bfloat162float(gate[(size_t)t * gate_stride + head0 + my_row]);
    const int set = warp / SET, part = warp % SET;
    auto together = [] { asm volatile("bar.sync 1, %0;" ::"n"(W * 32) : "memory"); };
    auto set_together = [&] { asm volatile("bar.sync %0, %1;" ::"r"(2 + set), "n"(SET * 32) : "memory"); };
    static_assert(D == 64 * SET && EK_PAGE == 16 * SET && STAGES % 2 == 0, "64 dimensions and 16 keys a warp; a set's stages");
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};   // rows g and g + 8; the sums of this thread's keys
    if (n_pages > 0) {
      // Q fragments of m16n8k16 for every 16-wide step of the head dimension: rows g and g + 8
      uint32_t qa[D / 16][4];
      const bf16* qrow = q + (size_t)t * q_row_stride + (size_t)head0 * D;
      const int a_row = (lane & 7) + 8 * ((lane >> 3) & 1);       // of an A fragment that ldmatrix fetches
      for (int idx = tid; idx < 16 * (D / 8); idx += W * 32) {
        const int r = idx / (D / 8), c = idx % (D / 8);
        const uint4 v = r < group ? *reinterpret_cast<const uint4*>(qrow + (size_t)r * D + 8 * c) : make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(q_s + r * (2 * D) + ((c ^ (r & 7)) << 4)) = v;
      }
      together();
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        ldsm_x4(smem_u32(q_s) + a_row * (2 * D) + (((2 * ks + (lane >> 4)) ^ (a_row & 7)) << 4), qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);
      together();                                  // (all have read the queries)
      // addresses are a lane's offset and a constant: 16-byte piece p of row r lies at (p ^ r) & 7
      const uint32_t ring = smem_u32(smem);
      const int k_row = 16 * part + (lane & 7) + 8 * (lane >> 4);
      const uint32_t key_at = k_row * 128 + ((((lane >> 3) & 1) ^ (k_row & 7)) << 4);
      const uint32_t value_at = part * kSub + a_row * 128 + (((lane >> 4) ^ (a_row & 7)) << 4);
      const uint32_t p_from = smem_u32(p_s) + set * 16 * 128, p_lower = smem_u32(q_s) - smem_u32(p_s), p_at = a_row * 128 + (((lane >> 4) ^ (a_row & 7)) << 4);
      unsigned char* const p_to = p_s + (16 * set + g) * 128 + 4 * tq;
      float* const max_to = max_s + set * 16 * SET + g * SET + part;
      const float4* const max_of = reinterpret_cast<const float4*>(max_s + set * 16 * SET + g * SET);
      const float by = cap.c > 0.f ? 1.f : scale_log2;
      int s = set, phase = 0;
      for (int i = set; i < n_pages; i += 2) {
        const int page0 = (pg_first + i) * EK_PAGE;
        const uint32_t stage = ring + s * kStage;
        float dot[2][2][4] = {};                 // [8 keys][even and odd steps of the head dimension]
        uint32_t kb[4][4];
        // ldmatrix x4: 16 keys x 16 dimensions a fetch, four steps ahead of their MMAs
        auto fetch_keys = [&](int ks) {
          ldsm_x4(stage + (ks >> 2) * kSub + (key_at ^ (32 * (ks & 3))), kb[ks & 3][0], kb[ks & 3][1], kb[ks & 3][2], kb[ks & 3][3]);
        };
        // (the warps meet in named barriers below: one that gave up goes on with them, and says so at the end)
        ok = ok && mbar_wait(full(s), phase, status, 42);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) fetch_keys(ks);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          mma_bf16_16816(dot[0][ks & 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[ks & 3][0], kb[ks & 3][1]);
          mma_bf16_16816(dot[1][ks & 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kb[ks & 3][2], kb[ks & 3][3]);
          if (ks + 4 < D / 16) fetch_keys(ks + 4);
        }
        // rows g (e < 2) and g + 8, keys 8u + 2tq + (e & 1) of the warp's
        float sc[2][4], mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[u][e] = (dot[u][0][e] + dot[u][1][e]) * by;
        if (cap.c > 0.f)
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[u][e] = capped_log2(sc[u][e], cap);
        const bool inside = page0 >= lo && page0 + EK_PAGE - 1 <= hi;
        if (!inside)
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int key = page0 + 16 * part + 8 * u + 2 * tq + (e & 1);
              if (key < lo || key > hi) sc[u][e] = -INFINITY;
            }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) mx[e >> 1] = fmaxf(mx[e >> 1], sc[u][e]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
          mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
        }
        if (tq == 0) {
          max_to[0] = mx[0];
          max_to[8 * SET] = mx[1];
        }
        set_together();
        float alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {            // (the maximum is finite from the first page on: it has a visible key)
          const float4 a = max_of[8 * r];
          const float m_new = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), m_run[r]);
          alpha[r] = ex2_approx(m_run[r] - m_new);
          m_run[r] = m_new;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float p0 = sc[u][2 * r] = ex2_approx(sc[u][2 * r] - m_new), p1 = sc[u][2 * r + 1] = ex2_approx(sc[u][2 * r + 1] - m_new);
            unsigned char* const to = p_to + 8 * r * 128 + (((2 * part + u) ^ (g & 7)) << 4);
            const uint32_t p = pack2_bf16(p0, p1);
            *reinterpret_cast<uint32_t*>(to) = p;
            *reinterpret_cast<uint32_t*>(to + (q_s - p_s)) = pack2_bf16(p0 - __uint_as_float(p << 16), p1 - __uint_as_float(p & 0xffff0000u));
          }
          l_run[r] = l_run[r] * alpha[r] + ((sc[0][2 * r] + sc[0][2 * r + 1]) + (sc[1][2 * r] + sc[1][2 * r + 1]));
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          acc[n][0] *= alpha[0]; acc[n][1] *= alpha[0];
          acc[n][2] *= alpha[1]; acc[n][3] *= alpha[1];
        }
        set_together();
        // both terms of P of 16 keys and their rows (which are keys and values alike), fetched a step ahead of their MMAs
        uint32_t pa[2][4], pb[2][4], vb[4][4];
        auto fetch_p = [&](int k) {
          const uint32_t from = p_from + (p_at ^ (32 * k));
          ldsm_x4(from, pa[k & 1][0], pa[k & 1][1], pa[k & 1][2], pa[k & 1][3]);
          ldsm_x4(from + p_lower, pb[k & 1][0], pb[k & 1][1], pb[k & 1][2], pb[k & 1][3]);
        };
        auto fetch_v = [&](int k, int x) {
          ldsm_x4_trans(stage + 16 * k * 128 + (value_at ^ (32 * x)), vb[x][0], vb[x][1], vb[x][2], vb[x][3]);
        };
        auto add = [&](int k, int x0) {          // to 32 dimensions: four sums in turn
#pragma unroll
          for (int term = 0; term < 2; ++term) {
            const uint32_t (&p)[4] = term == 0 ? pa[k & 1] : pb[k & 1];
#pragma unroll
            for (int x = x0; x < x0 + 2; ++x) {
              mma_bf16_16816(acc[2 * x], p[0], p[1], p[2], p[3], vb[x][0], vb[x][1]);
              mma_bf16_16816(acc[2 * x + 1], p[0], p[1], p[2], p[3], vb[x][2], vb[x][3]);
            }
          }
        };
        if (inside) {
          fetch_p(0);
#pragma unroll
          for (int x = 0; x < 4; ++x) fetch_v(0, x);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (k < 3) fetch_p(k + 1);
#pragma unroll
            for (int x = 0; x < 4; x += 2) {
              add(k, x);
              if (k < 3) fetch_v(k + 1, x);
              if (k < 3) fetch_v(k + 1, x + 1);
            }
          }
        } else {
          // at the edge of what is visible: steps without a visible key stay out of it (their rows may hold anything)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (page0 + 16 * k <= hi && page0 + 16 * k + 15 >= lo) {
              fetch_p(k);
#pragma unroll
              for (int x = 0; x < 4; ++x) fetch_v(k, x);
#pragma unroll
              for (int x = 0; x < 4; x += 2) add(k, x);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty(s));
        s += 2;
        if (s >= STAGES) {
          s -= STAGES;
          phase ^= 1;
        }
      }
    }
    // ---------------------------------------------------------- the two sets, merged; then the splits, in order
    // A warp keeps 32 of its dimensions, the first half in set 0 and the second in set 1, and has those of the other set's
    // warp added to them.  The pages are all consumed: the ring is dead.
    together();
    float* const o_s = (float*)smem;             // [warp][16 heads][32 dimensions], rows 40 apart for the banks
    constexpr int OS = 40;
    static_assert((size_t)W * 16 * OS * 4 <= (size_t)STAGES * kStage, "the exchange must fit the ring");
    float kept[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      float* const to = o_s + (warp * 16 + g) * OS + 8 * n + 2 * tq;
      *reinterpret_cast<float2*>(to) = set ? make_float2(acc[n][0], acc[n][1]) : make_float2(acc[n + 4][0], acc[n + 4][1]);
      *reinterpret_cast<float2*>(to + 8 * OS) = set ? make_float2(acc[n][2], acc[n][3]) : make_float2(acc[n + 4][2], acc[n + 4][3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) kept[n][e] = set ? acc[n + 4][e] : acc[n][e];
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
      if (tq == 0) {
        max_s[(set * 16 + g + 8 * r) * SET + part] = l_run[r];
        if (part == 0) row_s[set * 16 + g + 8 * r] = m_run[r];
      }
    }
    together();
    float l[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = g + 8 * r, other = set ^ 1;
      const float m_other = row_s[other * 16 + row], m = fmaxf(m_run[r], m_other);
      const float f = m_run[r] == -INFINITY ? 0.f : exp2f(m_run[r] - m);       // (a set without a page)
      const float f_other = m_other == -INFINITY ? 0.f : exp2f(m_other - m);
      auto sum_of = [&](int of) {
        const float4 x = *reinterpret_cast<const float4*>(max_s + (of * 16 + row) * SET);
        return (x.x + x.y) + (x.z + x.w);
      };
      const float l_own = sum_of(set) * f, l_other = sum_of(other) * f_other;
      l[r] = set ? l_other + l_own : l_own + l_other;
      m_run[r] = m;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float2 x = *reinterpret_cast<const float2*>(o_s + ((other * SET + part) * 16 + row) * OS + 8 * n + 2 * tq);
        kept[n][2 * r] = kept[n][2 * r] * f + x.x * f_other;
        kept[n][2 * r + 1] = kept[n][2 * r + 1] * f + x.y * f_other;
      }
    }
    const int dim0 = 64 * part + 32 * set + 2 * tq;
    // a sink: one more term exp(sink) in the denominator, with no value (-inf: none), counted once
    auto sink_of = [&](int r) { return sinks ? sinks[head0 + r] * 1.4426950408889634f : sink_log2; };   // per head, if given
    auto with_sink = [&](float sum, float m, float sk) { return sk > -INFINITY && sum > 0.f ? sum + exp2f(sk - m) : sum; };
    // a gated head's output is multiplied by the sigmoid of its gate
    auto gate_of = [&](int r) { return gate == nullptr ? 1.f : __bfloat162float(gate[(size_t)t * gate_stride + head0 + r]); };
    auto opened = [&](float x) { return gate == nullptr ? 1.f : 1.f / (1.f + expf(-x)); };
    auto value = [](float o, float sum, float by) { return (sum == 0.f ? 0.f : o / sum) * by; };     // (NaN stays NaN)
    bf16* o_t = out + ((size_t)t * n_q_heads + head0) * D;
    if (n_splits == 1) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int row = g + 8 * r;
        if (row >= group || !ok) continue;
        const float sum = with_sink(l[r], m_run[r], sink_of(row)), by = opened(gate_of(row));
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          bf16* to = o_t + (size_t)row * D + dim0 + 8 * n;
          const float x = value(kept[n][2 * r], sum, by), y = value(kept[n][2 * r + 1], sum, by);
          *reinterpret_cast<uint32_t*>(to) = pack2_bf16(x, y);
        }
      }
    } else {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      const float per_run = 1.f / (float)run;    // (idx / run exactly: both are below 2^13)
      if (ok) {                                  // (what a block that gave up does not send, the others wait for in vain)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int row = g + 8 * r;
          if (row >= group) continue;
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            const int idx = row * D + dim0 + 8 * n, owner = (int)(((float)idx + 0.5f) * per_run);
            st_async_f32x2(&recv_o[split * run + idx - owner * run], (unsigned)owner, make_float2(kept[n][2 * r], kept[n][2 * r + 1]), received);
          }
          if (tq == 0)
            for (int sp = warp; sp < n_splits; sp += W)        // every block needs this head's maximum and sum
              st_async_f32x2(&recv_ml[(split * 16 + row) * 2], (unsigned)sp, make_float2(m_run[r], l[r]), received);
        }
      }
      ok = ok && mbar_wait(received, 0, status, 43);
      if (ok)
        for (int slot = 4 * tid; slot < mine; slot += 4 * W * 32) {
          const int idx = split * run + slot, row = idx / D;
          float m = -INFINITY;
          for (int sp = 0; sp < n_splits; ++sp) m = fmaxf(m, recv_ml[(sp * 16 + row) * 2]);
          float sum = 0.f;
          float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int sp = 0; sp < n_splits; ++sp) {
            const float ls = recv_ml[(sp * 16 + row) * 2 + 1];
            if (ls != 0.f) {                     // else that split held no visible key
              const float f = exp2f(recv_ml[(sp * 16 + row) * 2] - m);
              const float4 v = *reinterpret_cast<const float4*>(recv_o + sp * run + slot);
              sum += ls * f;
              o.x += v.x * f; o.y += v.y * f; o.z += v.z * f; o.w += v.w * f;
            }
          }
          if (slot != 4 * tid) {
            my_sink = sink_of(row);
            my_gate = gate_of(row);
          }
          sum = with_sink(sum, m, my_sink);
          const float by = opened(my_gate);
          bf16* to = o_t + idx;
          const float x[4] = {value(o.x, sum, by), value(o.y, sum, by), value(o.z, sum, by), value(o.w, sum, by)};
          *reinterpret_cast<uint2*>(to) = make_uint2(pack2_bf16(x[0], x[1]), pack2_bf16(x[2], x[3]));
        }
    }
  }
  const int failed = __syncthreads_or(ok ? 0 : 1);
  if (failed)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);     // let copies in flight land
  if (n_splits > 1) cluster_sync();              // no block leaves while a sum may still be on its way to it
}

// DEEP: a ring twice as deep (192 KB, one block an SM) for launches that leave SMs empty anyway, so
// that more of a block's pages are on their way before the wait returns.  (Rows of 256 have the deep
// ring only: two blocks' registers would not fit an SM.)
template <int D, bool DEEP, bool QUERY = false>
static int launch_dt(bf16* out, const bf16* q, int q_row_stride, const int* positions,
                     const int* token_slot, const void* k_pages, const void* v_pages,
                     long long page_rows, const int* block_table, int table_stride, int n_tokens,
                     int n_q_heads, int n_kv_heads, float scale, int window, int n_splits, int* status,
                     float sink, const float* sinks, int chunk, float softcap, const bf16* gate, int gate_stride, cudaStream_t stream) {
  constexpr bool SHARED = D == 256;
  static_assert(!SHARED || DEEP, "rows of 256: the deep ring only");
  constexpr int STAGES = (D >= 128 ? 3 : 6) * (DEEP ? 2 : 1);
  constexpr int DB = D / 64;
  constexpr size_t smem = 1024 + (size_t)STAGES * (SHARED ? 1 : 2) * DB * EK_PAGE * 128 + (2 * STAGES + (SHARED ? 2 : 0)) * 8 +
                          (size_t)(kDtRecvO<D> + kDtRecvMl + (SHARED ? kDtWarps<D> * 16 + 2 * 16 : 0)) * 4 +
                          (SHARED ? 2 * 16 * 128 + 16 * D * 2 : 0);
  CUtensorMap mk, mv;
  int rc;
  if (!QUERY) {
    if ((rc = tensor_map(k_pages, page_rows, D, D, EK_PAGE, &mk))) return rc;
    if (!SHARED && (rc = tensor_map(v_pages, page_rows, D, D, EK_PAGE, &mv))) return rc;
  }
  const auto kernel = [] {
    if constexpr (SHARED) return attention_decode_tma_shared_kernel<D, STAGES>;
    else return attention_decode_tma_kernel<D, STAGES>;
  }();
  static bool configured[kMaxDevices] = {};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  if (device < 0 || device >= kMaxDevices) return EK_ERR_ARG;
  if (!configured[device]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    if (!DEEP || SHARED) {                       // clusters of 9 to 16 blocks
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return (int)e;
    }
    configured[device] = true;
  }
  prefer_carveout((const void*)kernel, 100);
  dim3 grid(n_splits, SHARED ? n_kv_heads * ((n_q_heads / n_kv_heads + 15) / 16) : n_kv_heads, n_tokens);
  if (QUERY) {                                   // can a cluster of 16 of these blocks run at all?
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kDtMaxSplits, 1, 1);
    cfg.blockDim = dim3(kDtThreads<D>);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kDtMaxSplits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) { cudaGetLastError(); return 0; }
    return clusters;
  }
  const float log2e = 1.4426950408889634f;
  const SoftCap cap = soft_cap(scale, softcap);
  auto launch = [&](auto... args) {
    if (n_splits > 1)
      return (int)launch_pdl_cluster_x(kernel, grid, dim3(kDtThreads<D>), smem, stream, n_splits, args...);
    return (int)launch_pdl(kernel, grid, dim3(kDtThreads<D>), smem, stream, args...);
  };
  if constexpr (SHARED)
    return launch(out, q, q_row_stride, positions, token_slot, mk, block_table, table_stride, n_kv_heads, n_q_heads,
                  scale * log2e, window, status, sink * log2e, sinks, chunk, cap, gate, gate_stride);
  else
    return launch(out, q, q_row_stride, positions, token_slot, mk, mv, block_table, table_stride, n_kv_heads, n_q_heads,
                  scale * log2e, window, status, sink * log2e, sinks, chunk, cap);
}

}  // namespace ek

// How many blocks may share a token on this device: 16 if clusters of that size can be
// scheduled for this head size, else 8 (0: the head size has no such kernel).
EK_EXPORT int ek_attention_decode_tma_max_splits(int head_dim) {
  using namespace ek;
  int clusters = 0;
  if (head_dim == 64)
    clusters = launch_dt<64, false, true>(nullptr, nullptr, 0, nullptr, nullptr, &clusters, &clusters, 64,
                                          nullptr, 0, 1, 1, 1, 1.f, 0, 1, nullptr, -INFINITY, nullptr, 0, 0.f, nullptr, 0, nullptr);
  else if (head_dim == 128)
    clusters = launch_dt<128, false, true>(nullptr, nullptr, 0, nullptr, nullptr, &clusters, &clusters, 64,
                                           nullptr, 0, 1, 1, 1, 1.f, 0, 1, nullptr, -INFINITY, nullptr, 0, 0.f, nullptr, 0, nullptr);
  else if (head_dim == 256)
    clusters = launch_dt<256, true, true>(nullptr, nullptr, 0, nullptr, nullptr, &clusters, &clusters, 64,
                                          nullptr, 0, 1, 1, 1, 1.f, 0, 1, nullptr, -INFINITY, nullptr, 0, 0.f, nullptr, 0, nullptr);
  else
    return 0;
  return clusters >= 1 ? kDtMaxSplits : kDtPortableSplits;
}

// head_dim 64 or 128 with at most 16 query heads a KV head, or 256 with k_pages == v_pages; 1 to 16 splits (each takes whole pages of
// the token's visible range); q rows 4-byte aligned; n_pages = pages in k_pages / v_pages
// ([pages, kv heads, 64, head_dim]); `status` is one int on the device.  `sink`: score of a key
// without a value that every query also sees (one more term in the softmax denominator);
// -INFINITY for none; `sinks` (may be null): one such score per query head, in place of `sink`.
// `chunk` > 0 instead of a window: keys of the token's own chunk of positions only.
// `softcap` > 0: scores become softcap tanh(score / softcap).  `gate` (null but for rows of 256): a value per token
// and query head (rows `gate_stride` apart) whose sigmoid the head's output is multiplied by.
EK_EXPORT int ek_attention_decode_tma(void* out, const void* q, int q_row_stride,
                                      const int* positions, const int* token_slot,
                                      const void* k_pages, const void* v_pages, int n_pages,
                                      const int* block_table, int table_stride, int n_tokens,
                                      int n_q_heads, int n_kv_heads, int head_dim, float scale,
                                      int window, int n_splits, int* status, float sink,
                                      const float* sinks, int chunk, float softcap, const void* gate,
                                      int gate_stride, cudaStream_t stream) {
  using namespace ek;
  if (n_tokens <= 0) return 0;
  if (chunk < 0 || (chunk > 0 && window > 0)) return EK_ERR_ARG;
  if ((head_dim != 64 && head_dim != 128 && head_dim != 256) || n_kv_heads <= 0 || n_q_heads % n_kv_heads ||
      (head_dim == 256 ? k_pages != v_pages || n_q_heads > 65535 : n_q_heads / n_kv_heads > 16) || n_splits < 1 || n_splits > kDtMaxSplits || q_row_stride % (head_dim == 256 ? 8 : 2) ||
      ((uintptr_t)q & (head_dim == 256 ? 15 : 3)) || (head_dim == 256 ? ((uintptr_t)out & 7) != 0 : gate != nullptr) || !status || n_kv_heads > 65535 || n_tokens > 65535 || n_pages <= 0)
    return EK_ERR_ARG;
  const long long page_rows = (long long)n_pages * n_kv_heads * EK_PAGE;
  // one block an SM at most, and a cluster of the portable size (a deep ring is one block an SM)
  const bool deep = (long long)n_tokens * n_kv_heads * n_splits <= sm_count() && n_splits <= kDtPortableSplits;
#define EK_DT(D_, DEEP_)                                                                          \
  return launch_dt<D_, DEEP_>((bf16*)out, (const bf16*)q, q_row_stride, positions, token_slot,     \
                              k_pages, v_pages, page_rows, block_table, table_stride, n_tokens,   \
                              n_q_heads, n_kv_heads, scale, window, n_splits, status, sink, sinks,     \
                              chunk, softcap, (const bf16*)gate, gate_stride, stream)
  if (head_dim == 256) EK_DT(256, true);
  if (head_dim == 64) {
    if (deep) EK_DT(64, true);
    EK_DT(64, false);
  }
  if (deep) EK_DT(128, true);
  EK_DT(128, false);
#undef EK_DT
}
