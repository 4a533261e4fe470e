// De-quantizer of 4-bit block-wise weights in the layout of bitsandbytes 0.43.2 (`functional.dequantize_4bit`,
// which the reference calls as `BF.dequantize_nf4(w, quant_state)`, models/utils/compute_utils.py:19, 29 and
// models/llama/fused_llama_layer_intra_inter_full_fuse.py:218-219, 359, 367, 379).  That library is not part of
// this build; what is restated here is its published storage format:
//   * two 4-bit codes per byte, the HIGH nibble first: element 2 i in bits 7..4 of byte i, element 2 i + 1 in bits 3..0;
//   * value = code_table[code] * absmax[element / blocksize], computed in fp32, rounded once to bf16;
//   * the 16-entry code table travels with the quant state (NF4 or FP4: whatever the table holds);
//   * "double quantization": absmax itself stored as 8-bit codes, absmax = table256[code] * absmax2[block / blocksize2]
//     + offset (fp32).
// A warp turns runs of 512 packed bytes into 1024 bf16 values with coalesced loads and stores; HBM-bound: 0.5 + 2
// bytes per element.  A launch takes up to four weights (the ones that the next product reads together), dealt out as one
// list of runs: each launch of its own ends with SMs idle.  Block numbers come from shifts (block sizes are powers of two;
// others divide): the 64-bit divisions were a quarter of the instructions.  The result is written with the default cache
// policy, the product behind it reads what fits from L2.
#include "hyc_common.cuh"

namespace hyc {

constexpr int kNf4Jobs = 4;
struct Nf4Job {
  const uint8_t* packed;
  const float *code16, *absmax;           // absmax null: nested
  const uint8_t* absmax_q;
  const float *code256, *absmax2;
  __nv_bfloat16* out;
  int64_t numel, first_run;               // runs of the jobs before
  int blocksize, blocksize2, shift, shift2;    // shift < 0: the block size is no power of two
  float offset;
};
struct Nf4Jobs { Nf4Job job[kNf4Jobs]; int count; int64_t runs; };

__device__ __forceinline__ float nf4_scale(const Nf4Job& j, int64_t e) {
  const int64_t blk = j.shift >= 0 ? e >> j.shift : e / j.blocksize;
  if (j.absmax) return j.absmax[blk];
  const int64_t blk2 = j.shift2 >= 0 ? blk >> j.shift2 : blk / j.blocksize2;
  // two roundings, as the library's two steps (block-wise de-quantization of the codes, then `+= offset`)
  return __fadd_rn(__fmul_rn(j.code256[j.absmax_q[blk]], j.absmax2[blk2]), j.offset);
}

__global__ void __launch_bounds__(256)
dequant_nf4_kernel(const __grid_constant__ Nf4Jobs jobs) {
  pdl_wait();
  __shared__ float s_code[kNf4Jobs][16];
  if (threadIdx.x < 16 * jobs.count) s_code[threadIdx.x >> 4][threadIdx.x & 15] = jobs.job[threadIdx.x >> 4].code16[threadIdx.x & 15];
  __syncthreads();
  // A warp takes runs of 1024 elements: four coalesced 128-byte loads (4 bytes = 8 elements per lane and load), four
  // coalesced 512-byte stores (16 bytes per lane and store).  All loads of a run are issued before the first use.
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < jobs.runs; r += n_warps) {
    int which = 0;
#pragma unroll
    for (int i = 1; i < kNf4Jobs; ++i)
      if (i < jobs.count && r >= jobs.job[i].first_run) which = i;
    const Nf4Job& j = jobs.job[which];
    const float* code = s_code[which];
    const int64_t e_run = (r - j.first_run) * 1024;
    const bool one_scale = (j.blocksize % 8) == 0;        // the 8 elements of a lane share a block
    uint32_t w[4];
    float s[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __ldcs(reinterpret_cast<const uint32_t*>(j.packed + e_run / 2) + 32 * i + lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = nf4_scale(j, e_run + 256 * i + 8 * lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t e0 = e_run + 256 * i + 8 * lane;
      uint32_t o[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const uint32_t byte = (w[i] >> (8 * b)) & 0xffu;
        const float s0 = one_scale ? s[i] : nf4_scale(j, e0 + 2 * b);
        const float s1 = one_scale ? s[i] : nf4_scale(j, e0 + 2 * b + 1);
        o[b] = pack_bf16x2_rn(__fmul_rn(code[byte >> 4], s0),           // element 2 b: the high nibble
                              __fmul_rn(code[byte & 15u], s1));         // element 2 b + 1
      }
      *reinterpret_cast<uint4*>(j.out + e0) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  // what is left of each tensor (fewer than 1024 elements): one element per thread of the first block
  if (blockIdx.x == 0) {
    for (int i = 0; i < jobs.count; ++i) {
      const Nf4Job& j = jobs.job[i];
      for (int64_t e = j.numel / 1024 * 1024 + threadIdx.x; e < j.numel; e += blockDim.x) {
        const uint32_t byte = j.packed[e >> 1];
        const uint32_t c = (e & 1) ? (byte & 15u) : (byte >> 4);
        j.out[e] = __float2bfloat16_rn(__fmul_rn(s_code[i][c], nf4_scale(j, e)));
      }
    }
  }
}

static int shift_of(int blocksize) {
  int s = 0;
  while ((1 << s) < blocksize && s < 30) ++s;
  return (1 << s) == blocksize ? s : -1;
}

}  // namespace hyc

using namespace hyc;

extern "C" HYC_API int hyc_dequant_nf4_many(int count, const hyc_nf4_job* in, void* stream) {
  if (!in) return HYC_ERR_NULL;
  if (count < 1 || count > kNf4Jobs) return HYC_ERR_SHAPE;
  Nf4Jobs jobs = {};
  int64_t total = 0;
  for (int i = 0; i < count; ++i) {
    const hyc_nf4_job& j = in[i];
    if (!j.packed || !j.code16 || !j.out) return HYC_ERR_NULL;
    const bool nested = j.absmax == nullptr;
    if (nested && (!j.absmax_q || !j.code256 || !j.absmax2)) return HYC_ERR_NULL;
    if (j.numel < 0 || j.blocksize <= 0 || (nested && j.blocksize2 <= 0)) return HYC_ERR_SHAPE;
    if (!aligned(j.packed, 4) || !aligned(j.out, 16)) return HYC_ERR_ALIGN;
    jobs.job[i] = {(const uint8_t*)j.packed, j.code16, j.absmax, j.absmax_q, j.code256, j.absmax2, (__nv_bfloat16*)j.out, j.numel, jobs.runs,
                   j.blocksize, nested ? j.blocksize2 : 1, shift_of(j.blocksize), nested ? shift_of(j.blocksize2) : 0, j.offset};
    jobs.runs += j.numel / 1024;
    total += j.numel;
  }
  jobs.count = count;
  if (total == 0) return HYC_OK;
  int64_t grid = (jobs.runs + 7) / 8;                 // one warp per run, eight warps per block
  const int64_t cap = (int64_t)num_sms() * 8;
  if (grid > cap) grid = cap;
  if (grid < 1) grid = 1;
  launch_pdl(dequant_nf4_kernel, dim3((unsigned)grid), dim3(256), 0, (cudaStream_t)stream, jobs);
  HYC_CHECK_LAUNCH();
  return HYC_OK;
}

extern "C" HYC_API int hyc_dequant_nf4(const void* packed, const float* code16, const float* absmax_f32,
                                       const uint8_t* absmax_q, const float* code256, const float* absmax2,
                                       int blocksize2, float offset, int64_t numel, int blocksize, void* out,
                                       void* stream) {
  const hyc_nf4_job job = {packed, code16, absmax_f32, absmax_q, code256, absmax2, out, numel, blocksize, blocksize2, offset};
  return hyc_dequant_nf4_many(1, &job, stream);
}
