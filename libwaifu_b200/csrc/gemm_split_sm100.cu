// One-round GEMM: products of so few tiles that the persistent kernel (gemm_sm100.cu) would leave
// most SMs idle or walk a long K with the few that have a tile.
//
// A CTA computes one 128 x block_n tile and leaves, so block_n is whatever multiple of 16 spreads
// the columns over the SMs, and where even that leaves SMs over, a cluster of 2, 4 or 8 CTAs
// divides the tile's K stages: each accumulates its share in its own tensor memory, writes the
// columns it does not own into their owners' shared memory (distributed shared memory), and
// finishes its own block_n / split columns: sum over the cluster in rank order, scale, bias, GELU,
// residual, one rounding. Nothing passes through global memory and no CTA waits for one that is
// not resident.
//   warps 0-7  an e4m3 weight against 16-bit rows: widen a stage's weight tile to the rows' type
//              (exact) into a two-slot ring of swizzled tiles; then, all kinds, the epilogue
//   warp  8    producer: TMA loads of the 128 rows and the weight tile of each K stage into a ring
//   warp  9    MMA: four tcgen05.mma per stage (128 x block_n, 32 bytes of K per row each)
// Every operand row of a stage is 128 bytes in the 128-byte swizzle, except the raw e4m3 tile of
// the widening form (64 bytes of K, as it lies).
//
// PAIR, for 16-bit rows of more than one row block: a cluster of two CTAs computes a tile of 256 rows with
// tcgen05.mma.cta_group::2, each with 128 of the rows and half of the tile's columns, which it loads,
// widens and keeps for both. So a weight tile is fetched and widened once for 256 rows, where the form
// above does it for 128. K stays in one piece.
#include "gemm_split_sm100.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "ptx_sm100.cuh"

namespace flsm100 {

namespace {

constexpr int kTileM = 128;
constexpr int kStageRowBytes = 128;
constexpr int kStepsPerStage = 4;  // 32 bytes of K per tcgen05.mma
constexpr int kWorkWarps = 8;
constexpr int kLoadWarp = kWorkWarps;
constexpr int kIssueWarp = kWorkWarps + 1;
constexpr int kSplitThreads = (kWorkWarps + 2) * 32;
constexpr int kMaxLoadStages = 8;
constexpr int kMaxWideSlots = 4;
constexpr int kATileBytes = kTileM * kStageRowBytes;
constexpr int kSmemPerCta = 227 * 1024 - 1024;  // (static shared memory beside it)

// A pair's estimate has to be this far below the other form's, or the persistent kernel's. Half rows of a short
// K in tiles above 128 columns are estimated too low by more: of 46 such shapes 14 lie between the two lines, and 13 of
// them measured slower in pairs (1593 x 1696 x 816 14.0 us in tiles of 128 rows and 15.0 in pairs, 1553 x 1856 x 672 13.7
// and 14.4, 569 x 4528 x 1088 15.9 and 16.6); below both lines 18.1 and 16.8 (2001 x 1632 x 1120).
constexpr float kPairMargin = 0.94f, kPairMarginShortHalf = 0.9f;
constexpr int kPairShortStages = 18;

struct SplitParams {
  int m, n, num_kb;
  int tiles_m;
  int split, block_n, cols;  // cols = block_n / split: what a CTA of the cluster finishes
  int load_stages, load_bytes, wide_off, wide_slots;
  const float *row_scale;
  const float *col_scale;
  int col_scale_scalar;
  const void *bias;
  const void *residual;
  int residual_rows;
  long long residual_ld;
  int act, is_bf16;
  void *out;
  int vector_io;  // out and the residual are 16-byte aligned with pitches of whole 16-byte pieces
  uint32_t tmem_cols;
  uint32_t *status;
};

// The exchange buffer holds groups of four columns, a group's 128 rows one after the other (so a
// warp's 32 rows leave as 512 contiguous bytes: sent row by row, 16 bytes each, 128 x 256 sums took
// their owners 14 us), groups 16 bytes more than that apart (so that readers of one row in
// neighbouring groups meet different banks).
constexpr int kGroupBytes = kTileM * 16 + 16;

__device__ __forceinline__ void store_v4(uint32_t addr, const uint32_t *v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

__device__ __forceinline__ void store_cluster_v4(uint32_t cluster_addr, const uint32_t *v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}

// Eight 16-bit values of one 16-byte piece added to x.
__device__ __forceinline__ void add8(float (&x)[8], const uint4 q, int is_bf16) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    if (is_bf16) {
      x[2 * h] += __uint_as_float(w[h] << 16);
      x[2 * h + 1] += __uint_as_float(w[h] & 0xffff0000u);
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[h]));
      x[2 * h] += f.x;
      x[2 * h + 1] += f.y;
    }
  }
}

__device__ __forceinline__ const uint16_t *residual_at(const SplitParams &p, int row, int col) {
  const int r = p.residual_rows == p.m ? row : row % p.residual_rows;
  return reinterpret_cast<const uint16_t *>(p.residual) + r * p.residual_ld + col;
}

__device__ __forceinline__ void prefetch_l2(const void *at) { asm volatile("prefetch.global.L2 [%0];" ::"l"(at)); }

// KIND: kKindF8, or kKindF16 / kKindBF16 with WIDEN: the weight is e4m3 and the rows are 16-bit.
template <int KIND, bool WIDEN, bool PAIR = false>
__global__ void __launch_bounds__(kSplitThreads, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const SplitParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  static_assert(WIDEN || !PAIR, "pairs are for the widening form");
  __shared__ __align__(8) uint64_t full_bar[kMaxLoadStages], empty_bar[kMaxLoadStages];
  __shared__ __align__(8) uint64_t raw_full_bar[PAIR ? kMaxLoadStages : 1];  // this CTA's share of the weight tile
  __shared__ __align__(8) uint64_t wide_full_bar[kMaxWideSlots], wide_empty_bar[kMaxWideSlots];
  __shared__ __align__(8) uint64_t acc_full_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile uint32_t abort_flag;

  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t lane = threadIdx.x & 31;
  // (a pair's CTAs finish all columns of their own rows, as an undivided tile's do)
  const int peer = PAIR ? static_cast<int>(cluster_cta_rank()) : 0;
  const int rank = !PAIR && p.split > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const bool leader = peer == 0;
  const int tile = blockIdx.x / (PAIR ? 2 : p.split);
  const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;  // neighbours share a weight tile
  const int m0 = PAIR ? (2 * tm + peer) * kTileM : tm * kTileM;
  const int n0 = tn * p.block_n;
  const int b_rows = PAIR ? p.block_n / 2 : p.block_n;  // of the weight tile, in this CTA
  const int b_row0 = n0 + peer * b_rows;
  const int kb0 = p.num_kb * rank / p.split, kb1 = p.num_kb * (rank + 1) / p.split;
  const int b_row_bytes = WIDEN ? kStageRowBytes / 2 : kStageRowBytes;

  if (warp == 0) {
    if (static_cast<int>(lane) < p.load_stages) {
      mbar_init(&full_bar[lane], 1);
      mbar_init(&empty_bar[lane], 1);
      if constexpr (PAIR) mbar_init(&raw_full_bar[lane], 1);
    }
    if (lane < kMaxWideSlots) {
      mbar_init(&wide_full_bar[lane], WIDEN ? kWorkWarps / p.wide_slots * (PAIR ? 2 : 1) : 1);
      mbar_init(&wide_empty_bar[lane], 1);
    }
    if (lane == 0) {
      abort_flag = 0;
      mbar_init(&acc_full_bar, 1);
    }
    fence_barrier_init();
  }
  if (warp == kLoadWarp && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    // The first stages of the weight into L2 while the kernel ahead in the stream may still run: a
    // prefetch writes nothing and the loads below read what they would have read anyway.
    for (int kb = kb0; kb < kb1 && kb < kb0 + p.load_stages; ++kb) tma_prefetch_l2_2d(&tmap_b, kb * b_row_bytes, b_row0);
  }
  if (warp == kIssueWarp) {
    tmem_alloc<PAIR ? 2 : 1>(&tmem_base_slot, p.tmem_cols);
    tmem_relinquish<PAIR ? 2 : 1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // the other CTA's barriers exist before anything signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  griddep_wait();
  griddep_launch_dependents();

  // The residual of the rows this CTA will finish, into L2 under the main loop.
  if (p.residual && warp < kWorkWarps) {
    const int lines = (p.cols * 2 + 127) / 128, first_col = n0 + rank * p.cols;
    for (int i = static_cast<int>(threadIdx.x); i < kTileM * lines; i += kWorkWarps * 32) {
      const int row = m0 + i / lines, col = first_col + i % lines * 64;
      if (row < p.m && col < p.n) prefetch_l2(residual_at(p, row, col));
    }
  }

  if (warp == kLoadWarp) {
    if (elect_one()) {
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      const uint32_t bytes = static_cast<uint32_t>(kATileBytes + p.block_n * b_row_bytes);  // (rows outside arrive as zeros)
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[s], phase ^ 1, &abort_flag)) {
          ok = false;
          break;
        }
        uint8_t *base = smem + s * p.load_bytes;
        if constexpr (PAIR) {
          // The weight's bytes count on this CTA's own barrier, for its widening warps, the rows of both
          // CTAs on the leader's.
          mbar_arrive_expect_tx(&raw_full_bar[s], static_cast<uint32_t>(b_rows * b_row_bytes));
          tma_load_2d(base + kATileBytes, &tmap_b, &raw_full_bar[s], kb * b_row_bytes, b_row0);
          if (leader) mbar_arrive_expect_tx(&full_bar[s], 2 * kATileBytes);
          tma_load_2d_pair(base, &tmap_a, map_to_cta(smem_u32(&full_bar[s]), 0), kb * kStageRowBytes, m0);
        } else {
          mbar_arrive_expect_tx(&full_bar[s], bytes);
          tma_load_2d(base + kATileBytes, &tmap_b, &full_bar[s], kb * b_row_bytes, n0);
          tma_load_2d(base, &tmap_a, &full_bar[s], kb * kStageRowBytes, m0);
        }
        if (++s == p.load_stages) {
          s = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        abort_flag = 1;
        atomicCAS(p.status, 0u, static_cast<uint32_t>(kStatusProducerTimeout));
      }
    }
  } else if (warp == kIssueWarp) {
    // (the whole warp walks the loop and one lane issues, as in the persistent kernel)
    // A pair's leader issues for both; its commits arrive at the same barrier in both.
    const bool issuer = elect_one();
    constexpr uint32_t kFmt = KIND == kKindBF16 ? 1u : 0u;
    const uint32_t idesc = umma_idesc(PAIR ? 2 * kTileM : kTileM, static_cast<uint32_t>(p.block_n), kFmt, kFmt);
    const uint32_t smem0 = smem_u32(smem);
    auto commit = [&](uint64_t *bar) {
      if constexpr (PAIR) {
        umma_commit_pair_both(bar);
      } else {
        umma_commit(bar);
      }
    };
    bool ok = true;
    int s = 0, w = 0;
    uint32_t phase = 0, wide_phase = 0;
    for (int kb = leader ? kb0 : kb1; kb < kb1; ++kb) {
      if (!mbar_wait(&full_bar[s], phase, &abort_flag) || (WIDEN && !mbar_wait(&wide_full_bar[w], wide_phase, &abort_flag))) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint64_t ad = umma_desc_sw128(smem0 + s * p.load_bytes);
      const uint64_t bd = umma_desc_sw128(WIDEN ? smem0 + p.wide_off + w * b_rows * kStageRowBytes
                                                : smem0 + s * p.load_bytes + kATileBytes);
#pragma unroll
      for (int i = 0; i < kStepsPerStage; ++i) {
        if constexpr (PAIR) {
          if (issuer) umma_ss_pair<KIND>(tmem_base, ad + i * 2, bd + i * 2, idesc, (kb > kb0 || i > 0) ? 1u : 0u);
        } else {
          if (issuer) umma_ss<KIND>(tmem_base, ad + i * 2, bd + i * 2, idesc, (kb > kb0 || i > 0) ? 1u : 0u);
        }
      }
      if (issuer) {
        commit(&empty_bar[s]);
        if (WIDEN) commit(&wide_empty_bar[w]);
      }
      if (WIDEN && ++w == p.wide_slots) {
        w = 0;
        wide_phase ^= 1;
      }
      if (++s == p.load_stages) {
        s = 0;
        phase ^= 1;
      }
    }
    if (ok && issuer && leader) commit(&acc_full_bar);
    if (!ok && issuer) {
      abort_flag = 1;
      atomicCAS(p.status, 0u, static_cast<uint32_t>(kStatusMmaTimeout));
    }
  } else if constexpr (WIDEN) {
    // Sixteen e4m3 bytes of a row -> two 16-byte pieces of its 128 bytes, in the 128-byte swizzle.
    // The warps share out the wide slots (several stages are widened at once), and the load stages are
    // a multiple of those, so that a warp sees every phase of the barriers it waits on.
    const int group_warps = kWorkWarps / p.wide_slots;
    const int w = static_cast<int>(warp) / group_warps;
    const int first = static_cast<int>(threadIdx.x) % (group_warps * 32);
    bool ok = true;
    for (int it = w; it < kb1 - kb0; it += p.wide_slots) {
      const int s = it % p.load_stages;
      if (!mbar_wait(PAIR ? &raw_full_bar[s] : &full_bar[s], (it / p.load_stages) & 1, &abort_flag) ||
          !mbar_wait(&wide_empty_bar[w], ((it / p.wide_slots) & 1) ^ 1, &abort_flag)) {
        ok = false;
        break;
      }
      const uint8_t *raw = smem + s * p.load_bytes + kATileBytes;
      uint8_t *wide = smem + p.wide_off + w * b_rows * kStageRowBytes;
#pragma unroll 4
      for (int piece = first; piece < b_rows * 4; piece += group_warps * 32) {
        const uint32_t r = static_cast<uint32_t>(piece) >> 2, q = static_cast<uint32_t>(piece) & 3;
        const uint4 v = *reinterpret_cast<const uint4 *>(raw + piece * 16);
        uint4 lo, hi;
        if constexpr (KIND == kKindBF16) {
          e4m3x16_to_bf16(v, &lo, &hi);
        } else {
          e4m3x16_to_f16(v, &lo, &hi);
        }
        uint8_t *row_base = wide + r * kStageRowBytes;
        *reinterpret_cast<uint4 *>(row_base + (((2 * q) ^ (r & 7)) << 4)) = lo;
        *reinterpret_cast<uint4 *>(row_base + (((2 * q + 1) ^ (r & 7)) << 4)) = hi;
      }
      fence_proxy_async_smem();  // the UMMA reads these bytes through the async proxy
      __syncwarp();
      if (lane == 0) {
        if (PAIR && !leader) {
          mbar_arrive_remote(map_to_cta(smem_u32(&wide_full_bar[w]), 0));
        } else {
          mbar_arrive(&wide_full_bar[w]);
        }
      }
    }
    if (!ok && lane == 0) {
      abort_flag = 1;
      atomicCAS(p.status, 0u, static_cast<uint32_t>(kStatusProducerTimeout));
    }
  }

  // ------------------------------------------------------------------ epilogue
  // The accumulator is complete: so are all loads and all reads of the ring, which becomes the
  // exchange buffer: split x 128 rows of `cols` floats, the part of every CTA of the cluster.
  bool have = false;
  if (warp < kWorkWarps) {
    have = __all_sync(0xffffffffu, mbar_wait(&acc_full_bar, 0, &abort_flag));
    if (!have && lane == 0) {
      abort_flag = 1;
      atomicCAS(p.status, 0u, static_cast<uint32_t>(kStatusEpilogueTimeout));
    }
  }
  // (The cluster barriers are reached on every path: all waits above are bounded.)
  if (p.split > 1) {
    __syncwarp();
    cluster_sync_all();
  }
  if (have) {
    tc_fence_after_sync();
    const uint32_t quarter = warp & 3;
    const int row = static_cast<int>(quarter) * 32 + static_cast<int>(lane);
    const uint32_t t_row = tmem_base + ((quarter * 32u) << 16);
    const uint32_t mine = smem_u32(smem) + static_cast<uint32_t>(rank * (p.cols / 4) * kGroupBytes + row * 16);
    for (int c = static_cast<int>(warp >> 2); c < p.block_n / 16; c += 2) {
      uint32_t v[16];
      tmem_ld_32x16(t_row + c * 16, v);
      tmem_ld_wait(v);
      const int owner = c * 16 / p.cols;
      const uint32_t local = mine + static_cast<uint32_t>((c * 16 - owner * p.cols) / 4) * kGroupBytes;
      if (owner == rank) {
#pragma unroll
        for (int j = 0; j < 4; ++j) store_v4(local + j * kGroupBytes, v + 4 * j);
      } else {
        const uint32_t dst = map_to_cta(local, static_cast<uint32_t>(owner));
#pragma unroll
        for (int j = 0; j < 4; ++j) store_cluster_v4(dst + j * kGroupBytes, v + 4 * j);
      }
    }
  }
  __syncwarp();
  if (p.split > 1) {
    cluster_sync_all();
  } else {
    __syncthreads();
  }
  if (have) {
    // A thread keeps its eight columns and walks the rows, so scales and bias are fetched once, and
    // the residual of four rows is on its way before the first is needed.
    const int groups = p.cols / 8, rows_at_once = kWorkWarps * 32 / groups;
    const int g = static_cast<int>(threadIdx.x) % groups, r0 = static_cast<int>(threadIdx.x) / groups;
    const int col = n0 + rank * p.cols + g * 8;
    const int live_rows = (r0 < rows_at_once && col < p.n) ? min(kTileM, p.m - m0) : 0;  // (n is a multiple of 8)
    float cs[8], bias[8];
    if (live_rows > 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        cs[i] = p.col_scale ? __ldg(p.col_scale + (p.col_scale_scalar ? 0 : col + i)) : 1.0f;
        bias[i] = 0.0f;
      }
      if (p.bias) {
        uint4 q;
        uint16_t *e = reinterpret_cast<uint16_t *>(&q);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = __ldg(reinterpret_cast<const uint16_t *>(p.bias) + col + i);
        add8(bias, q, p.is_bf16);
      }
    }
    constexpr int kAhead = 4;
    for (int r = r0; r < live_rows; r += kAhead * rows_at_once) {
      uint4 res[kAhead];
      float rs[kAhead];
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int row = m0 + r + a * rows_at_once;
        res[a] = make_uint4(0, 0, 0, 0);
        rs[a] = 1.0f;
        if (r + a * rows_at_once >= live_rows) continue;
        if (p.row_scale) rs[a] = __ldg(p.row_scale + row);
        if (p.residual) {
          const uint16_t *at = residual_at(p, row, col);
          if (p.vector_io) {
            res[a] = *reinterpret_cast<const uint4 *>(at);
          } else {
            uint16_t *e = reinterpret_cast<uint16_t *>(&res[a]);
#pragma unroll
            for (int i = 0; i < 8; ++i) e[i] = at[i];
          }
        }
      }
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        const int in_tile = r + a * rows_at_once;
        if (in_tile >= live_rows) break;
        const uint8_t *part = smem + g * 2 * kGroupBytes + in_tile * 16;
        float x[8] = {};
        for (int s = 0; s < p.split; ++s, part += p.cols / 4 * kGroupBytes) {
          const float4 lo = *reinterpret_cast<const float4 *>(part), hi = *reinterpret_cast<const float4 *>(part + kGroupBytes);
          x[0] += lo.x, x[1] += lo.y, x[2] += lo.z, x[3] += lo.w, x[4] += hi.x, x[5] += hi.y, x[6] += hi.z, x[7] += hi.w;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] *= rs[a] * cs[i];
        if (p.bias) {
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] += bias[i];
        }
        if (p.act == kActGeluTanh) {
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = gelu_tanh(x[i]);
        }
        if (p.residual) add8(x, res[a], p.is_bf16);
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          if (p.is_bf16) {
            const __nv_bfloat162 q = __floats2bfloat162_rn(x[2 * h], x[2 * h + 1]);
            w[h] = *reinterpret_cast<const uint32_t *>(&q);
          } else {
            const __half2 q = __floats2half2_rn(x[2 * h], x[2 * h + 1]);
            w[h] = *reinterpret_cast<const uint32_t *>(&q);
          }
        }
        uint16_t *dst = reinterpret_cast<uint16_t *>(p.out) + static_cast<long long>(m0 + in_tile) * p.n + col;
        if (p.vector_io) {
          *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) dst[i] = static_cast<uint16_t>(i & 1 ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu);
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (abort_flag != 0) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // copies that may still be in flight
    __syncthreads();
  }
  // The leader's instructions read the other CTA's shared memory, and both signal each other.
  if constexpr (PAIR) cluster_sync_all();
  if (warp == kIssueWarp) {
    tc_fence_after_sync();
    tmem_dealloc<PAIR ? 2 : 1>(tmem_base, p.tmem_cols);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      return reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return static_cast<EncodeTiledFn>(nullptr);
  }();
  return fn;
}

// A (rows, row_bytes) byte matrix read in boxes of box_bytes x box_rows, zeros outside.
bool make_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t row_bytes, uint32_t box_bytes, uint32_t box_rows,
              CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {row_bytes, rows};
  cuuint64_t strides[1] = {row_bytes};
  cuuint32_t box[2] = {box_bytes, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// What a launch makes of a plan; host arithmetic only.
struct SplitGeometry {
  int num_kb, tiles_m, ctas;
  int load_bytes, load_stages, wide_slots, wide_off;
  int smem_bytes;
};

SplitGeometry split_geometry(bool widen, int m, int n, int k, const SplitPlan &plan) {
  SplitGeometry g = {};
  const int tile_m = plan.pair ? 2 * kTileM : kTileM, b_rows = plan.pair ? plan.block_n / 2 : plan.block_n;
  g.num_kb = (k * (widen ? 2 : 1) + kStageRowBytes - 1) / kStageRowBytes;
  g.tiles_m = (m + tile_m - 1) / tile_m;
  g.ctas = g.tiles_m * ((n + plan.block_n - 1) / plan.block_n) * (plan.pair ? 2 : plan.split);
  g.load_bytes = kATileBytes + b_rows * (widen ? kStageRowBytes / 2 : kStageRowBytes);
  g.wide_slots = b_rows <= (plan.pair ? 96 : 128) ? kMaxWideSlots : 2;
  const int wide_bytes = widen ? g.wide_slots * b_rows * kStageRowBytes : 0;
  const int longest = (g.num_kb + plan.split - 1) / plan.split;
  g.load_stages = std::min((kSmemPerCta - 1024 - wide_bytes) / g.load_bytes, kMaxLoadStages);
  if (widen) {
    g.load_stages -= g.load_stages % g.wide_slots;
  } else {
    g.load_stages = std::min(g.load_stages, longest);
  }
  g.wide_off = g.load_stages * g.load_bytes;
  const int exchange = plan.block_n / 4 * kGroupBytes;
  g.smem_bytes = std::max(g.wide_off + wide_bytes, exchange) + 1024;
  return g;
}

template <int KIND, bool WIDEN, bool PAIR = false>
cudaError_t launch_split(const GemmArgs &a, const SplitPlan &plan, const char **why) {
  const uint64_t row_bytes = static_cast<uint64_t>(a.k) * (KIND == kKindF8 ? 1 : 2);
  CUtensorMap ta, tb;
  const uint32_t bn = static_cast<uint32_t>(PAIR ? plan.block_n / 2 : plan.block_n);  // weight rows to a CTA
  if (!make_map(&ta, a.a, a.m, row_bytes, kStageRowBytes, kTileM, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !(WIDEN ? make_map(&tb, a.b, a.n, row_bytes / 2, kStageRowBytes / 2, bn, CU_TENSOR_MAP_SWIZZLE_NONE)
              : make_map(&tb, a.b, a.n, row_bytes, kStageRowBytes, bn, CU_TENSOR_MAP_SWIZZLE_128B))) {
    *why = "cuTensorMapEncodeTiled refused an operand";
    return cudaErrorInvalidValue;
  }
  auto kernel = gemm_split_kernel<KIND, WIDEN, PAIR>;
  static bool attr_set = false;  // per instantiation
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta);
    if (e != cudaSuccess) {
      *why = "cudaFuncSetAttribute(max dynamic shared memory) failed";
      return e;
    }
    attr_set = true;
  }
  SplitParams p = {};
  p.m = a.m;
  p.n = a.n;
  const SplitGeometry g = split_geometry(WIDEN, a.m, a.n, a.k, plan);
  p.num_kb = g.num_kb;
  p.tiles_m = g.tiles_m;
  p.split = plan.split;
  p.block_n = plan.block_n;
  p.cols = plan.block_n / plan.split;
  p.load_bytes = g.load_bytes;
  p.wide_slots = g.wide_slots;
  p.load_stages = g.load_stages;
  p.wide_off = g.wide_off;
  p.row_scale = a.row_scale;
  p.col_scale = a.col_scale;
  p.col_scale_scalar = a.col_scale_scalar;
  p.bias = a.bias;
  p.residual = a.residual;
  p.residual_rows = a.residual_rows > 0 ? a.residual_rows : a.m;
  p.residual_ld = a.residual_ld;
  p.act = a.act;
  p.is_bf16 = a.out_bf16;
  p.out = a.out;
  p.vector_io = (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 &&
                (!a.residual || ((reinterpret_cast<uintptr_t>(a.residual) & 15) == 0 && a.residual_ld % 8 == 0));
  p.tmem_cols = 32;
  while (p.tmem_cols < static_cast<uint32_t>(plan.block_n)) p.tmem_cols *= 2;
  p.status = a.status;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(g.ctas), 1, 1);
  cfg.blockDim = dim3(kSplitThreads, 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(g.smem_bytes);
  cfg.stream = a.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(PAIR ? 2 : plan.split);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = PAIR || plan.split > 1 ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ta, tb, p);
  if (e != cudaSuccess) *why = "kernel launch failed";
  return e;
}

}  // namespace

bool gemm_split_supported(const GemmArgs &a) {
  if (a.num_extra_out > 0 || a.row_amax || a.rows_per_group || a.global_scale) return false;
  if (a.out_ld > 0 && (a.out_ld != a.n || a.out_col0 != 0)) return false;
  return encode_fn() != nullptr;
}

// Estimated times in microseconds, fitted to a sweep of every block_n and split over 1280 to 16384
// channels, k = 640 to 12288 and 16 to 2048 rows. A stage takes its latency, or its bytes through L2 with
// every CTA pulling at once, or (widening) what the converters need for block_n rows; then come the
// exchange and the epilogue, which grow with block_n, and the launch.
//   77 x 2560 x 2048, half: 17.7 us on the persistent kernel, 11.2 here; 300 x 1280 x 640 15.4 and
//   7.8; 512 x 5120 x 3072 in bfloat16 39 (with a widening pass) and 30.7; e4m3 rows with
//   the quantiser, 300 x 1280 x 1280 15.3 and 10.0, 1024 x 3072 x 3072 21.8 and 20.1.
static SplitPlan timed_plan(GemmKind kind, int b_is_e4m3, int m, int n, int k, int sms, bool stream_k, float *estimate) {
  SplitPlan best = {0, 0, false};
  *estimate = 0.0f;
  if (kind != kGemmE4M3 && !b_is_e4m3) return best;
  const bool widen = kind != kGemmE4M3;
  const int num_kb = (k * (widen ? 2 : 1) + kStageRowBytes - 1) / kStageRowBytes;
  const int tiles_m = (m + kTileM - 1) / kTileM;
  // The linears on quantised rows give the same bits with and without the rows' maxima, to one destination
  // and to several, in row groups and without; some of those forms run on the persistent kernel alone.
  // So e4m3 rows stay there wherever that kernel cuts a tile's K in two (260 x 9488 x 5376), and keep K in
  // one piece here (10.9 -> 12.4 us at 128 x 3072 x 3072, still below 13.8).
  if (!widen && stream_k) {
    int tile_plan[8];
    gemm_plan(kind, m, n, k, sms, 1, tile_plan);
    if (tile_plan[6] > 0) return best;
  }
  // The persistent kernel: rounds of whole tiles (pairs of CTAs above one row block), a long K cut in
  // halves where that leaves no unit without one (gemm_schedule; its other cut, of the tail of more
  // tiles, is not priced: 16-bit rows measured 0.63 to 0.98 of it here), and for bfloat16 rows the pass
  // that widens the weight ahead of it. e4m3 rows, whose K is never divided here, leave a K that the
  // other kernel halves to it, whether or not it may (512 x 3072 x 12288: 36.6 us there, 39.8 here; whole
  // on both sides, 38.2 and 35.7, but 212 x 6736 x 11440 44.1 and 49.9).
  const int units = tiles_m == 1 ? sms : sms / 2;
  const long long tiles = tiles_m == 1 ? (n + 127) / 128 : static_cast<long long>((m + 255) / 256) * ((n + 255) / 256);
  float persistent = static_cast<float>((tiles + units - 1) / units * num_kb) *
                     (tiles_m == 1 ? (widen ? 0.23f : 0.19f) : (widen ? 0.31f : 0.35f));
  if (2 * tiles <= units && num_kb >= 80) {
    if (!widen) return best;
    persistent *= 0.75f;
  }
  persistent += tiles_m == 1 ? 10.0f : 12.8f;
  if (kind == kGemmBF16) persistent += static_cast<float>(n) * k * 0.65e-6f;
  // Where the two kernels' measured times cross, over some 300 shapes of each kind with estimates from 0.75
  // to 1.2 of each other and weights that come from HBM. Half: the persistent kernel takes 1.12 of its
  // estimate, this one 0.98, so products up to a tenth above it come here (216 x 11544 x 1280: estimates
  // 19.4 and 19.0, measured 17.6 here, 21.9 there). bfloat16: 1.06 and 1.00 up to k = 2048, 1.01 and 1.02
  // to 4096, 0.96 and 1.05 beyond (1547 x 2024 x 2912, estimates 33.9 and 30.9, measured 35.5 and 33.3),
  // but not where the widened copy it reads is 100 MB and no longer in L2 (367 x 8792 x 11296 132 us there,
  // 108 here).
  // e4m3 rows whose pitch is no multiple of a 32-byte sector cost a fifth sector per 128 bytes, and tiles
  // of 128 rows read a long K more often than the persistent kernel's of 256 (1342 x 1672: 37.2 us here and
  // 33.8 there at k = 7120, 26.9 and 29.3 at 7104), unless that one needs a second round.
  // Taken and more than 2 % slower are 2, 4 and 8 of those shapes.
  float margin = 1.0f;
  if (kind == kGemmF16) margin = 1.1f;
  if (kind == kGemmBF16) {
    margin = static_cast<int64_t>(n) * k < 50'000'000 ? std::max(0.7f, 1.1f - 3.5e-5f * static_cast<float>(k)) : 1.0f;
  }
  if (!widen && k % 32 != 0 && num_kb > 32 && tiles_m > 1 && tiles <= units) margin = 0.85f;
  float best_time = persistent * margin;
  const int max_split = widen ? 8 : 1;
  for (int split = 1; split <= max_split; split *= 2) {
    // clusters of four and eight do not fill every SM of a GPC
    const int room = split <= 2 ? sms : split == 4 ? sms * 9 / 10 : sms * 3 / 4;
    if (num_kb < 2 * split) break;
    const int step = 16 * split;
    for (int bn = std::max(32, step); bn <= 256; bn += step) {
      const long long ctas = static_cast<long long>(tiles_m) * ((n + bn - 1) / bn) * split;
      if (ctas > room) continue;
      const float bytes = kATileBytes + bn * (widen ? kStageRowBytes / 2 : kStageRowBytes);
      const float through_l2 = ctas * bytes / (widen ? 8.0e6f : 12.5e6f);
      const float stage = std::max(std::max(widen ? 0.39f : 0.215f, through_l2), bn * (widen ? 0.0023f : 0.0016f));
      const float exchange = split == 1 ? 0.0f : split == 2 ? 1.1f : split == 4 ? 2.3f : 4.7f;
      const float scale = split == 1 ? 1.0f : split == 2 ? 0.707f : split == 4 ? 0.5f : 0.354f;
      const float time = (num_kb + split - 1) / split * stage + bn * scale * (widen ? 0.044f : 0.03f) + exchange + (widen ? 2.6f : 6.3f);
      if (time < best_time) {
        best_time = time;
        best = {bn, split, false};
      }
    }
  }
  *estimate = best_time;
  return best;
}

SplitPlan gemm_split_plan(GemmKind kind, int b_is_e4m3, int m, int n, int k, int sms, bool stream_k) {
  float estimate;
  return timed_plan(kind, b_is_e4m3, m, n, k, sms, stream_k, &estimate);
}

// Estimated as above, fitted to 34 shapes of 129 to 2048 rows, each at every width: a stage takes its way through
// the widening warps and across the pair and back, 0.315 us with four widened slots, 0.45 with two, which tiles
// above 192 columns have (four would leave four slots of the load ring, which is whole turns of the other). 512 x
// 5120 x 3072 in bfloat16: 30.6 us in tiles of 128 rows, 25.1 in tiles of 256 x 160; 238 x 14088 x 2304 31.1 and 23.4,
// 1705 x 1400 x 3696 in half 34.5 and 27.6; below some thirty tiles the shorter stages and the divided K of the other
// form win (300 x 2560 x 2048 15.9 and 16.9). Of 119 products drawn at random that it takes, half rows are 9 % faster on
// average and bfloat16 rows 11 %, and three more than 2 % slower (310 x 7040 x 1200: 17.1 and 18.4, a second row block
// that is nearly empty).
SplitPlan gemm_pair_plan(GemmKind kind, int m, int n, int k, int sms) {
  SplitPlan best = {0, 0, false};
  if ((kind != kGemmF16 && kind != kGemmBF16) || m <= kTileM || gemm_single_cta_only()) return best;
  float other, best_time = 0.0f;
  timed_plan(kind, 1, m, n, k, sms, true, &other);
  const int num_kb = (k * 2 + kStageRowBytes - 1) / kStageRowBytes;
  const int tiles_m = (m + 2 * kTileM - 1) / (2 * kTileM);
  for (int bn = 64; bn <= 256; bn += 32) {
    if (static_cast<long long>(tiles_m) * ((n + bn - 1) / bn) > sms / 2) continue;
    const float time = num_kb * (bn <= 192 ? 0.315f : 0.45f) + bn * 0.029f + (bn <= 192 ? 5.2f : 5.8f);
    const bool short_half = kind == kGemmF16 && num_kb <= kPairShortStages && bn > 128;
    if (time < other * (short_half ? kPairMarginShortHalf : kPairMargin) && (best.split == 0 || time < best_time)) {
      best_time = time;
      best = {bn, 1, true};
    }
  }
  return best;
}

namespace {

void describe(bool widen, int m, int n, int k, const SplitPlan &cut, int *plan) {
  for (int i = 0; i < 8; ++i) plan[i] = 0;
  if (cut.split == 0) return;
  const SplitGeometry g = split_geometry(widen, m, n, k, cut);
  plan[0] = cut.block_n, plan[1] = cut.split, plan[2] = g.ctas, plan[3] = g.num_kb;
  plan[4] = g.load_stages, plan[5] = widen ? g.wide_slots : 0, plan[6] = g.load_bytes, plan[7] = g.smem_bytes;
}

}  // namespace

void gemm_split_describe(GemmKind kind, int m, int n, int k, int sms, bool stream_k, int *plan) {
  describe(kind != kGemmE4M3, m, n, k, gemm_split_plan(kind, kind != kGemmE4M3, m, n, k, sms, stream_k), plan);
}

void gemm_pair_describe(GemmKind kind, int m, int n, int k, int sms, int *plan) {
  describe(true, m, n, k, gemm_pair_plan(kind, m, n, k, sms), plan);
}

cudaError_t launch_gemm_split(const GemmArgs &a, const SplitPlan &plan, const char **why) {
  *why = "";
  switch (a.kind) {
    case kGemmE4M3: return launch_split<kKindF8, false>(a, plan, why);
    case kGemmBF16: return plan.pair ? launch_split<kKindBF16, true, true>(a, plan, why) : launch_split<kKindBF16, true>(a, plan, why);
    default: return plan.pair ? launch_split<kKindF16, true, true>(a, plan, why) : launch_split<kKindF16, true>(a, plan, why);
  }
}

}  // namespace flsm100
