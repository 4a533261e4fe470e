// Host entry of the split GEMM kernels (tc_split.cu).
#pragma once
#include "tc_common.cuh"

namespace hyc {
namespace tc {

// split > 0: launch with the split kernels, the pair form (256-row tiles) if `pair`; split = 0: the persistent kernel
// A frozen weight as 4-bit block-wise codes (the format: nf4.cu), decoded on its way into a product of up to 128 rows.  Element e is
// code16[nibble e] * absmax[e >> shift], rounded once to bf16; absmax null: two-level, as there.  packed null: the operand is bf16
struct FourView {
  const uint8_t* packed;
  const float *code16, *absmax;
  const uint8_t* absmax_q;
  const float *code256, *absmax2;
  int64_t ld;                               // elements of a row
  int shift, shift2;
  float offset;
};
struct FourWeights { FourView w[4]; };      // as the B operands: K segments or weights side by side
bool four_pays(int epi, const Params& p, bool recorded);
int launch_four(int epi, int q_bit, bool b_mn, const Operands& ops, const Params& p, const FourWeights& four, cudaStream_t st);

struct SplitPlan { int split; bool pair; };
SplitPlan choose_split(int epi, const Params& p);
int launch_split(int epi, int q_bit, bool b_mn, const SplitPlan& plan, const Operands& ops, const Params& p, cudaStream_t st);

}  // namespace tc
}  // namespace hyc
