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
// bytes per element.  Where 16 columns share a scale and the tensors are aligned for it, a lane takes 16 elements at a time
// (8 bytes in, 32 out, two scales per run), and the next run's codes and scales are on their way while this one is written.  Two weights
// of 11008 x 4096: 51 us before (eight elements per lane, each run waiting for a chain of three loads), 41 now.  A launch takes up to four weights (the ones that the next product reads together), dealt out as one
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
  bool wide;                              // 16 elements share a scale, packed 8-byte and out 32-byte aligned
};
struct Nf4Jobs { Nf4Job job[kNf4Jobs]; int count; int64_t runs; };

__device__ __forceinline__ int64_t nf4_block(const Nf4Job& j, int64_t e) { return j.shift >= 0 ? e >> j.shift : e / j.blocksize; }
__device__ __forceinline__ int64_t nf4_block2(const Nf4Job& j, int64_t blk) { return j.shift2 >= 0 ? blk >> j.shift2 : blk / j.blocksize2; }
// two roundings, as the library's two steps (block-wise de-quantization of the codes, then `+= offset`)
__device__ __forceinline__ float nf4_nested(float code, float absmax2, float offset) { return __fadd_rn(__fmul_rn(code, absmax2), offset); }
__device__ __forceinline__ float nf4_scale(const Nf4Job& j, int64_t e) {
  const int64_t blk = nf4_block(j, e);
  if (j.absmax) return j.absmax[blk];
  return nf4_nested(j.code256[j.absmax_q[blk]], j.absmax2[nf4_block2(j, blk)], j.offset);
}

// what a lane needs for its two pieces of 16 elements of a run
struct Nf4Pieces {
  uint2 w[2];
  float a[2];                             // absmax, or the second-level factor of a nested one
  uint32_t q[2];                          // nested: its code
};
__device__ __forceinline__ void nf4_fetch(const Nf4Job& j, int64_t e_run, int lane, Nf4Pieces& p) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int64_t e = e_run + 512 * i + 16 * lane, blk = nf4_block(j, e);
    p.w[i] = ld_stream_v2(j.packed + e / 2);
    p.q[i] = 0u;
    if (j.absmax) {
      p.a[i] = j.absmax[blk];
    } else {
      p.q[i] = j.absmax_q[blk];
      p.a[i] = j.absmax2[nf4_block2(j, blk)];
    }
  }
}

__global__ void __launch_bounds__(256)
dequant_nf4_kernel(const __grid_constant__ Nf4Jobs jobs) {
  pdl_wait();
  __shared__ float s_code[kNf4Jobs][16];
  if (threadIdx.x < 16 * jobs.count) s_code[threadIdx.x >> 4][threadIdx.x & 15] = jobs.job[threadIdx.x >> 4].code16[threadIdx.x & 15];
  __syncthreads();
  // A warp takes runs of 1024 elements.
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  auto job_of = [&](int64_t r) {
    int which = 0;
#pragma unroll
    for (int i = 1; i < kNf4Jobs; ++i)
      if (i < jobs.count && r >= jobs.job[i].first_run) which = i;
    return which;
  };
  int next_job = 0;
  Nf4Pieces next = {};
  auto fetch = [&](int64_t r) {
    if (r >= jobs.runs) return;
    next_job = job_of(r);
    const Nf4Job& j = jobs.job[next_job];
    if (j.wide) nf4_fetch(j, (r - j.first_run) * 1024, lane, next);
  };
  fetch(warp);
  for (int64_t r = warp; r < jobs.runs; r += n_warps) {
    const int which = next_job;
    const Nf4Pieces cur = next;
    fetch(r + n_warps);
    const Nf4Job& j = jobs.job[which];
    const float* code = s_code[which];
    const int64_t e_run = (r - j.first_run) * 1024;
    if (j.wide) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float s = j.absmax ? cur.a[i] : nf4_nested(__ldg(j.code256 + cur.q[i]), cur.a[i], j.offset);
        uint32_t o[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const uint32_t byte = ((b < 4 ? cur.w[i].x : cur.w[i].y) >> (8 * (b & 3))) & 0xffu;
          o[b] = pack_bf16x2_rn(__fmul_rn(code[byte >> 4], s), __fmul_rn(code[byte & 15u], s));      // the high nibble first
        }
        st_v8(j.out + e_run + 512 * i + 16 * lane, o);
      }
      continue;
    }
    // four coalesced 128-byte loads (4 bytes = 8 elements per lane and load), four coalesced 512-byte stores (16 bytes per
    // lane and store); all loads of a run are issued before the first use
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
                   j.blocksize, nested ? j.blocksize2 : 1, shift_of(j.blocksize), nested ? shift_of(j.blocksize2) : 0, j.offset,
                   j.blocksize % 16 == 0 && aligned(j.packed, 8) && aligned(j.out, 32)};
    jobs.runs += j.numel / 1024;
    total += j.numel;
  }
  jobs.count = count;
  if (total == 0) return HYC_OK;
  int64_t grid = (jobs.runs + 7) / 8;                 // one warp per run, eight warps per block
  const int64_t cap = (int64_t)num_sms() * resident_blocks(dequant_nf4_kernel, 256, 0, 4);
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
