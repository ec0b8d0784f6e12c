// Host-side interface of the one-round GEMM (gemm_split_sm100.cu): the products whose tiles all fit
// the GPU at once, of launch_gemm's operands and epilogue.
#pragma once

#include <cuda_runtime.h>

#include "gemm_sm100.cuh"

namespace flsm100 {

// How a product is cut: tiles of 128 rows x `block_n` columns, each computed by a cluster of
// `split` CTAs that divide its K stages, or (`pair`, split 1) tiles of 256 rows, each computed by a
// pair of CTAs. split == 0: the product stays with the persistent kernel.
struct SplitPlan {
  int block_n;
  int split;
  bool pair;
};

// Host arithmetic only; for e4m3 against e4m3, and (`b_is_e4m3`) 16-bit rows against an e4m3 weight
// that is widened in the kernel. `stream_k`: whether the persistent kernel may cut tiles in two (it has
// the workspace for it).
SplitPlan gemm_split_plan(GemmKind kind, int b_is_e4m3, int m, int n, int k, int sms, bool stream_k);

// The cut of 16-bit rows against an e4m3 weight into tiles of 256 rows, where that is estimated to be
// faster than gemm_split_plan's or the persistent kernel; split == 0: it is not.
SplitPlan gemm_pair_plan(GemmKind kind, int m, int n, int k, int sms);

// gemm_split_plan's with what a launch makes of it, all 0 without a plan: plan[8] is block_n, split, CTAs, K stages,
// ring slots, widened slots (16-bit rows), bytes of a ring slot, dynamic shared memory of a CTA.
void gemm_split_describe(GemmKind kind, int m, int n, int k, int sms, bool stream_k, int *plan);
void gemm_pair_describe(GemmKind kind, int m, int n, int k, int sms, int *plan);  // the same of gemm_pair_plan's

// Whether the kernel has all that `args` asks for (one destination of pitch n, no row groups, no
// row maxima).
bool gemm_split_supported(const GemmArgs &args);

cudaError_t launch_gemm_split(const GemmArgs &args, const SplitPlan &plan, const char **why);

}  // namespace flsm100
