// The experts' products for many tokens on pairs of SMs: tcgen05.mma.cta_group::2, the expert's weight rows
// on the 256-row side of the MMA and a tile of the plan - up to 256 (token, choice) pairs that chose the
// expert - on the other, as wide as the tile is (steps of 32).  A prompt spreads its pairs over the experts
// unevenly (2,048 tokens, 4 of 32 experts: about 256 +- 16 pairs each); with the pairs on the side of the
// MMA that takes any width, an expert's pairs are cut into few equal tiles and at most 31 rows a tile are
// padding, where fixed tiles of 128 pairs would leave a quarter of the work to padding.
//
// Structure of the pair product (gemm_pair_bf16.cu): a cluster of two blocks, each staging half of both
// operands (128 weight rows and half of the tile's pairs, 64 of K a stage, a ring of six stages whose copies
// complete on the first block's barrier); the first block's thread issues the MMAs for both; two
// accumulators of 256 columns, so that a tile's epilogue runs under the next tile's MMAs; the pairs of SMs
// walk the units (tile, 256 weight rows), a tile's units side by side so that its rows come from L2.
//   up    the tile's rows come gathered by token from x (one tile::gather4 copy a lane of the producer warp
//         brings four rows), or, with many pairs, from a copy of x in the plan's order (moe_gather in moe.cu):
//         gathered rows reach shared memory at half the rate of boxes
//   down  the tile's rows stand side by side: a box of 16 rows a lane
// A thread of the epilogue holds one weight row - one column of the result - for the tile's pairs, so a
// warp stores 32 neighbouring columns of a pair at once.  Gate and up rows alternate: neighbouring lanes
// exchange values, and each of the two forms every other pair's output.
// Every barrier wait is bounded, as there.
//
// Bound by the tensor pipe and the last round of units in a prompt, by the weights' way from memory in a decode
// step.  Measured (32 experts of 1,024 gated, width 2,048, 4 chosen; up + down, us; the mma.sync tiles of 64 x 128
// before): 2,048 tokens 296 + 170 -> 105 + 58 (up with the copy of its rows; 630 TFLOP/s of the chosen pairs' work),
// 8 tokens 60 + 34 -> 46 + 23 (21 experts chosen: 264 MB in 69 us).
#include "moe_common.cuh"
#include "tc_pair.cuh"

namespace ek {

constexpr int kMoeWRows = 128;                  // weight rows ONE block stages
constexpr int kMoeTile = 256;                   // weight rows of a unit; most pairs of a tile
constexpr int kMoeEven = 32;                    // widths of a tile: multiples of this
constexpr int kMoeStages = 6;
constexpr int kMoeThreads = 320;
constexpr int kMoeEpilogueWarps = 8;
constexpr int kMoeBoxRows = 16;                 // rows a copy of the down form
constexpr uint32_t kMoeHalfBytes = kMoeWRows * kTcBK * 2;
constexpr uint32_t kMoeStageBytes = 2 * kMoeHalfBytes;
constexpr size_t kMoeSmem = (size_t)kMoeStages * kMoeStageBytes + (2 * kMoeStages + 4) * 8 + 16;

struct MoePairParams {
  void* out;                // up: bfloat16 [sorted row][N or N / 2]; down: 32-bit [pair][N]
  const int* tiles;         // [n][3]: expert, first sorted row, rows
  const int* n_tiles;
  const int* sorted_pair;
  const float* pair_weight; // per pair, or null
  int top;                  // up: token of a pair = pair / top
  int N, K, P;
  int blocks_n;             // units a tile
  int act, gated;
  float limit;
  int* status;
};

// Four rows of a K-major matrix (one box of 64 values each) into four neighbouring 128-byte rows of this
// block's shared memory; the bytes complete on a barrier that may stand in the other block of the pair.
__device__ __forceinline__ void tma_gather4_pair(uint32_t dst, const CUtensorMap* map, int c0, int4 rows,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(rows.x), "r"(rows.y), "r"(rows.z), "r"(rows.w), "r"(bar_cluster_addr)
      : "memory");
}

template <bool UP, bool GATHER>
__global__ void __launch_bounds__(kMoeThreads, 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                const MoePairParams prm) {
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bars = (uint64_t*)(smem + (size_t)kMoeStages * kMoeStageBytes);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kMoeStages),
                 acc_full0 = smem_u32(bars + 2 * kMoeStages), acc_empty0 = smem_u32(bars + 2 * kMoeStages + 2);
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * kMoeStages + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const int pair0 = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

  if (tid == 0) {
    tma_prefetch_map(&map_x);
    tma_prefetch_map(&map_w);
    for (int s = 0; s < kMoeStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, 2 * kMoeEpilogueWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMoeEpilogueWarps) tmem_alloc_pair(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  bool ok = (smem_u32(smem) & 1023u) == 0;
  if (!ok && tid == 0) atomicCAS(prm.status, 0, 59);
  const int n_units = prm.n_tiles[0] * prm.blocks_n;
  const int k_blocks = (prm.K + kTcBK - 1) / kTcBK;
  auto width_of = [](int rows) { return (rows + kMoeEven - 1) / kMoeEven * kMoeEven; };

  if (warp == kMoeEpilogueWarps) {
    // ------------------------------------------------------------------ producer warp of this block's halves
    const uint32_t full_first = map_to_rank(full0, 0);
    int c = 0;
    for (int u = pair0; u < n_units && ok; u += n_pairs) {
      const int* tile = prm.tiles + 3 * (u / prm.blocks_n);
      const int expert = tile[0], row0 = tile[1], rows = tile[2], half = width_of(rows) / 2;
      const int w_row = expert * prm.N + u % prm.blocks_n * kMoeTile + (int)rank * kMoeWRows;
      int4 from = make_int4(0, 0, 0, 0);
      bool copies;
      if (GATHER) {                               // rows behind the tile's last repeat its first: never stored
        copies = lane < half / 4;
        const int at = (int)rank * half + lane * 4;
        auto token = [&](int i) { return prm.sorted_pair[row0 + (i < rows ? i : 0)] / prm.top; };
        if (copies) from = make_int4(token(at), token(at + 1), token(at + 2), token(at + 3));
      } else {
        copies = lane < half / kMoeBoxRows;
        from.x = row0 + (int)rank * half + lane * kMoeBoxRows;
      }
      const uint32_t tx = 2 * kMoeHalfBytes + (uint32_t)half * 2 * kTcBK * 2;
      for (int kb = 0; kb < k_blocks; ++kb, ++c) {
        const int s = c % kMoeStages;
        if (c >= kMoeStages) {
          ok = mbar_wait(empty0 + 8 * s, ((c / kMoeStages) & 1) ^ 1, prm.status, 51);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        }
        const uint32_t dst = smem_u32(smem + (size_t)s * kMoeStageBytes);
        if (lane == 0) {
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, tx);
          tma_load_2d_pair(dst, &map_w, kb * kTcBK, w_row, full_first + 8 * s);
        }
        if (copies) {
          if (GATHER) tma_gather4_pair(dst + kMoeHalfBytes + (uint32_t)lane * 512, &map_x, kb * kTcBK, from, full_first + 8 * s);
          else tma_load_2d_pair(dst + kMoeHalfBytes + (uint32_t)lane * kMoeBoxRows * 128, &map_x, kb * kTcBK, from.x,
                                full_first + 8 * s);
        }
      }
    }
  } else if (tid == 32 * (kMoeEpilogueWarps + 1) && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer (first block)
    const uint32_t stage0 = smem_u32(smem);
    int c = 0, i = 0;
    uint32_t ready = 0;
    for (int u = pair0; u < n_units && ok; u += n_pairs, ++i) {
      const int width = width_of(prm.tiles[3 * (u / prm.blocks_n) + 2]);
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(width >> 3) << 17) |
                             ((uint32_t)(kMoeTile >> 4) << 24);
      const int buf = i & 1;
      if (i >= 2) {
        ok = mbar_wait(acc_empty0 + 8 * buf, ((i >> 1) & 1) ^ 1, prm.status, 52);
        if (!ok) break;
        tc_fence_after();
      }
      const uint32_t acc = tmem_base + (uint32_t)(buf * kMoeTile);
      for (int kb = 0; kb < k_blocks; ++kb, ++c) {
        const int s = c % kMoeStages;
        if (!ready) {
          ok = mbar_wait(full0 + 8 * s, (c / kMoeStages) & 1, prm.status, 53);
          if (!ok) break;
        }
        tc_fence_after();
        const uint32_t base = stage0 + (uint32_t)s * kMoeStageBytes;
        ready = mma_stage_pair(acc, smem_desc_k_sw128(base), smem_desc_k_sw128(base + kMoeHalfBytes), idesc,
                               kb ? 1u : 0u, empty0 + 8 * s, full0 + 8 * ((c + 1) % kMoeStages),
                               ((c + 1) / kMoeStages) & 1);
      }
      if (!ok) break;
      tc_commit_pair(acc_full0 + 8 * buf);
    }
  } else if (warp < kMoeEpilogueWarps) {
    // ------------------------------------------------------------------ epilogue
    const uint32_t acc_empty_first = map_to_rank(acc_empty0, 0);
    const int quarter = warp & 3, side = warp >> 2;        // weight rows 32 quarter ..., half of the pairs
    int i = 0;
    for (int u = pair0; u < n_units && ok; u += n_pairs, ++i) {
      const int* tile = prm.tiles + 3 * (u / prm.blocks_n);
      const int row0 = tile[1], rows = tile[2], half = width_of(rows) / 2;
      const int first = side * half, mine = min(half, rows - first);      // this warp's pairs of the tile
      const int n = u % prm.blocks_n * kMoeTile + (int)rank * kMoeWRows + quarter * 32 + lane;
      // lane's share of the pairs' numbers and weights
      int pid[4];
      float pw[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        pid[q] = q * 32 + lane < mine ? prm.sorted_pair[row0 + first + q * 32 + lane] : 0;
        pw[q] = prm.pair_weight != nullptr && q * 32 + lane < mine ? prm.pair_weight[pid[q]] : 1.f;
      }
      const int buf = i & 1;
      ok = mbar_wait(acc_full0 + 8 * buf, (i >> 1) & 1, prm.status, 54);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after();
      const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kMoeTile + first);
      float v[128];
#pragma unroll
      for (int j = 0; j < 128; j += 16)
        if (j < half) tmem_ld16_nowait(acc + j, v + j);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty_first + 8 * buf);

      // (one activation's code at a time: 64 outputs a thread with every activation in each do not fit the
      // instruction cache and made the gated product twice as slow)
      auto store_gated = [&](auto value) {
        // lanes 2c, 2c + 1 hold gate and up of output column c: the even lane forms the even pairs' outputs
        const bool odd = lane & 1;
        bf16* o = (bf16*)prm.out + (size_t)(row0 + first + odd) * (prm.N / 2) + n / 2;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q * 32 >= mine) break;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float w = __shfl_sync(0xffffffffu, pw[q], j + odd);
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v[q * 32 + j] : v[q * 32 + j + 1], 1);
            const float own = odd ? v[q * 32 + j + 1] : v[q * 32 + j];
            const float r = value((odd ? other : own) * w, (odd ? own : other) * w);
            if (q * 32 + j + odd < mine && n < prm.N) o[(size_t)(q * 32 + j) * (prm.N / 2)] = __float2bfloat16_rn(r);
          }
        }
      };
      auto store_plain = [&](auto value) {
        bf16* o = (bf16*)prm.out + (size_t)(row0 + first) * prm.N + n;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q * 32 >= mine) break;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float w = __shfl_sync(0xffffffffu, pw[q], j);
            const float r = value(v[q * 32 + j] * w);
            if (q * 32 + j < mine && n < prm.N) o[(size_t)(q * 32 + j) * prm.N] = __float2bfloat16_rn(r);
          }
        }
      };
      if (UP && prm.gated) {
        if (prm.act == ACT_SILU) store_gated([](float g, float up) { return gated_value(g, up, ACT_SILU, 0.f); });
        else if (prm.act == ACT_CLAMPED)
          store_gated([&](float g, float up) { return gated_value(g, up, ACT_CLAMPED, prm.limit); });
        else if (prm.act == ACT_GELU_TANH)
          store_gated([](float g, float up) { return gated_value(g, up, ACT_GELU_TANH, 0.f); });
        else if (prm.act == ACT_RELU2) store_gated([](float g, float up) { return gated_value(g, up, ACT_RELU2, 0.f); });
        else store_gated([](float g, float up) { return g * up; });
      } else if (UP) {
        if (prm.act == ACT_RELU2) store_plain([](float z) { return activate(z, ACT_RELU2); });
        else if (prm.act == ACT_SILU) store_plain([](float z) { return activate(z, ACT_SILU); });
        else if (prm.act == ACT_GELU_TANH) store_plain([](float z) { return activate(z, ACT_GELU_TANH); });
        else store_plain([](float z) { return z; });
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q * 32 >= mine) break;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int p = __shfl_sync(0xffffffffu, pid[q], j);
            const float w = __shfl_sync(0xffffffffu, pw[q], j);
            if (q * 32 + j < mine && n < prm.N) ((float*)prm.out)[(size_t)p * prm.N + n] = v[q * 32 + j] * w;
          }
        }
      }
    }
  }

  const int failed = __syncthreads_or(ok ? 0 : 1);
  if (failed)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);      // let copies in flight land
  tc_fence_before();
  cluster_sync();
  if (warp == kMoeEpilogueWarps) tmem_dealloc_pair(tmem_base, 512);
}

template <bool UP, bool GATHER>
static int launch_moe_pair(const void* x, long long x_rows, const void* w, int n_experts, MoePairParams prm,
                           int max_tiles, cudaStream_t stream) {
  auto kernel = moe_pair_kernel<UP, GATHER>;
  static int pairs_that_fit[kMaxDevices] = {};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  if (device < 0 || device >= kMaxDevices) return EK_ERR_ARG;
  CUtensorMap mx, mw;
  int rc;
  if ((rc = tensor_map(x, x_rows, prm.K, prm.K, GATHER ? 1 : kMoeBoxRows, &mx))) return rc;
  if ((rc = tensor_map(w, (long long)n_experts * prm.N, prm.K, prm.K, kMoeWRows, &mw))) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kMoeThreads);
  cfg.dynamicSmemBytes = kMoeSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  if (pairs_that_fit[device] == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMoeSmem);
    if (e != cudaSuccess) return (int)e;
    prefer_carveout((const void*)kernel, 100);
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) return (int)e;
    if (clusters < 1) return EK_ERR_ARG;
    pairs_that_fit[device] = clusters;
  }
  prm.blocks_n = (prm.N + kMoeTile - 1) / kMoeTile;
  const long long units = (long long)max_tiles * prm.blocks_n;
  if (units > (1ll << 30)) return EK_ERR_ARG;
  cfg.gridDim = dim3(2 * (unsigned)(units < pairs_that_fit[device] ? units : pairs_that_fit[device]));
  cfg.numAttrs = 2;
  return (int)cudaLaunchKernelEx(&cfg, kernel, mx, mw, prm);
}

static bool moe_pair_args(const void* x, const void* w, int N, int K, int n_experts, int max_tiles, const int* status) {
  return N > 0 && K > 0 && K % 8 == 0 && n_experts > 0 && status && max_tiles >= 0 && ((uintptr_t)x & 15) == 0 &&
         ((uintptr_t)w & 15) == 0 && (long long)n_experts * N < (1ll << 31);
}

}  // namespace ek

// `gathered`: x holds a row per pair in the plan's order (n_rows pairs) instead of one per token (n_rows tokens).
EK_EXPORT int ek_moe_pair_up(void* out, const void* x, const void* w, const int* tiles, const int* n_tiles,
                             const int* sorted_pair, int n_rows, int gathered, int n_experts, int max_tiles, int top, int N, int K,
                             int act, int gated, float limit, const float* row_weight, int* status,
                             cudaStream_t stream) {
  using namespace ek;
  if (max_tiles <= 0 || n_rows <= 0) return 0;
  if (!moe_pair_args(x, w, N, K, n_experts, max_tiles, status) || top <= 0 || (gated && N % 2) ||
      (act == ACT_CLAMPED && !(gated && limit > 0.f)))
    return EK_ERR_ARG;
  MoePairParams prm{};
  prm.out = out; prm.tiles = tiles; prm.n_tiles = n_tiles; prm.sorted_pair = sorted_pair;
  prm.pair_weight = row_weight; prm.top = top; prm.N = N; prm.K = K;
  prm.act = act; prm.gated = gated; prm.limit = limit; prm.status = status;
  return gathered ? launch_moe_pair<true, false>(x, n_rows, w, n_experts, prm, max_tiles, stream)
                  : launch_moe_pair<true, true>(x, n_rows, w, n_experts, prm, max_tiles, stream);
}

EK_EXPORT int ek_moe_pair_down(float* out, const void* a, const void* w, const int* tiles, const int* n_tiles,
                               const int* sorted_pair, const float* pair_weight, int n_rows, int n_experts,
                               int max_tiles, int N, int K, int* status, cudaStream_t stream) {
  using namespace ek;
  if (max_tiles <= 0 || n_rows <= 0) return 0;
  if (!moe_pair_args(a, w, N, K, n_experts, max_tiles, status)) return EK_ERR_ARG;
  MoePairParams prm{};
  prm.out = out; prm.tiles = tiles; prm.n_tiles = n_tiles; prm.sorted_pair = sorted_pair;
  prm.pair_weight = pair_weight; prm.top = 1; prm.N = N; prm.K = K; prm.status = status;
  return launch_moe_pair<false, false>(a, n_rows, w, n_experts, prm, max_tiles, stream);
}
