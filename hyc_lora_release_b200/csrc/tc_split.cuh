// Host entry of the split GEMM kernels (tc_split.cu).
#pragma once
#include "tc_common.cuh"

namespace hyc {
namespace tc {

// split > 0: launch with the split kernels, the pair form (256-row tiles) if `pair`; split = 0: the persistent kernel
struct SplitPlan { int split; bool pair; };
SplitPlan choose_split(int epi, const Params& p);
int launch_split(int epi, int q_bit, bool b_mn, const SplitPlan& plan, const Operands& ops, const Params& p, cudaStream_t st);

}  // namespace tc
}  // namespace hyc
