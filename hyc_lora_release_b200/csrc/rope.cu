// Rotary position embedding (rotate-half form) on the hidden layout [rows, n_heads * head_dim], the
// operation the fused layer applies to q and k after their projections and re-applies in the backward pass
// to the reconstructed q and k (models/llama/fused_llama_layer_intra_inter_full_fuse.py:142-143, 441, 449,
// 459-460 call rope_forward / rope_backward of operators/rope_kernels.py).
//
//   position p = row % seq_len,  h = head_dim / 2,  c = cos[p, j],  s = sin[p, j]   (j < h: the tables
//   repeat their first half in the second)
//   out[j]     = x[j] * c - x[j + h] * s
//   out[j + h] = x[j + h] * c + x[j] * s            backward: the same with s negated
//
// Arithmetic: that of the reference's kernel, which computes in the dtype of the sine table
// (operators/rope_kernels.py:73-78: `Q1 = tl.load(...).to(sin1.dtype)`): with bf16 tables every product and the
// sum are bf16 operations (three roundings per output); with fp32 tables they are separate fp32 operations and the
// store rounds to bf16.  No multiply-add contraction in either form.
// One thread owns eight adjacent j of one head: two 16-byte loads and two 16-byte stores of x, 16 (bf16
// tables) or 2 x 32 (fp32 tables) bytes of each table; the tables stay in L1/L2 (seq_len * head_dim values).
// Bound by memory.  Blocks are laid out over (octets of a row, rows), so that no index needs a 64-bit division, and a
// launch takes up to two tensors with the same rows (q and k of a layer).
#include "hyc_common.cuh"

namespace hyc {

struct RopeTensor { const __nv_bfloat16* x; __nv_bfloat16* out; int64_t ldx, ldo; int heads; };

template <bool TABLE_F32>
__global__ void __launch_bounds__(256)
rope_kernel(const RopeTensor t0, const RopeTensor t1, const void* __restrict__ cos_t, const void* __restrict__ sin_t, int64_t ld_table,
            int64_t rows, int seq_len, int head_dim, float sin_sign) {
  pdl_wait();
  const int half = head_dim >> 1;
  const int per_head = half >> 3;                       // octets of j per head
  const int w = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  int head = w / per_head;
  const int j0 = (w - head * per_head) << 3;
  if (head >= t0.heads + t1.heads) return;
  const bool second = head >= t0.heads;
  if (second) head -= t0.heads;
  const int64_t ldx = second ? t1.ldx : t0.ldx, ldo = second ? t1.ldo : t0.ldo;
  const __nv_bfloat16* __restrict__ x = (second ? t1.x : t0.x) + (int64_t)head * head_dim + j0;
  __nv_bfloat16* __restrict__ out = (second ? t1.out : t0.out) + (int64_t)head * head_dim + j0;
  for (int64_t row = blockIdx.y; row < rows; row += gridDim.y) {
    const int pos = (int)((uint32_t)row % (uint32_t)seq_len);      // rows < 2^32: checked by the caller
    const __nv_bfloat16* xp = x + row * ldx;
    const uint4 a = *reinterpret_cast<const uint4*>(xp);
    const uint4 b = *reinterpret_cast<const uint4*>(xp + half);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
    uint32_t o1[4], o2[4];
    if (TABLE_F32) {
      float c[8], s[8];
      const float* cp = reinterpret_cast<const float*>(cos_t) + pos * ld_table + j0;
      const float* sp = reinterpret_cast<const float*>(sin_t) + pos * ld_table + j0;
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        const float4 cv = *reinterpret_cast<const float4*>(cp + e), sv = *reinterpret_cast<const float4*>(sp + e);
        c[e] = cv.x; c[e + 1] = cv.y; c[e + 2] = cv.z; c[e + 3] = cv.w;
        s[e] = sv.x; s[e + 1] = sv.y; s[e + 2] = sv.z; s[e + 3] = sv.w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x1l = bf16lo_to_f32(aw[e]), x1h = bf16hi_to_f32(aw[e]);
        const float x2l = bf16lo_to_f32(bw[e]), x2h = bf16hi_to_f32(bw[e]);
        const float sl = s[2 * e] * sin_sign, sh = s[2 * e + 1] * sin_sign;
        const float cl = c[2 * e], ch = c[2 * e + 1];
        o1[e] = pack_bf16x2_rn(__fsub_rn(__fmul_rn(x1l, cl), __fmul_rn(x2l, sl)), __fsub_rn(__fmul_rn(x1h, ch), __fmul_rn(x2h, sh)));
        o2[e] = pack_bf16x2_rn(__fadd_rn(__fmul_rn(x2l, cl), __fmul_rn(x1l, sl)), __fadd_rn(__fmul_rn(x2h, ch), __fmul_rn(x1h, sh)));
      }
    } else {
      const uint4 cv = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(cos_t) + pos * ld_table + j0);
      const uint4 sv = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(sin_t) + pos * ld_table + j0);
      const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w}, sw[4] = {sv.x, sv.y, sv.z, sv.w};
      const uint32_t flip = sin_sign < 0.f ? 0x80008000u : 0u;     // backward: the sine negated (exact)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t sn = sw[e] ^ flip;
        const __nv_bfloat162 x1 = *reinterpret_cast<const __nv_bfloat162*>(&aw[e]);
        const __nv_bfloat162 x2 = *reinterpret_cast<const __nv_bfloat162*>(&bw[e]);
        const __nv_bfloat162 c2 = *reinterpret_cast<const __nv_bfloat162*>(&cw[e]);
        const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(&sn);
        const __nv_bfloat162 r1 = __hsub2_rn(__hmul2_rn(x1, c2), __hmul2_rn(x2, s2));
        const __nv_bfloat162 r2 = __hadd2_rn(__hmul2_rn(x2, c2), __hmul2_rn(x1, s2));
        o1[e] = *reinterpret_cast<const uint32_t*>(&r1);
        o2[e] = *reinterpret_cast<const uint32_t*>(&r2);
      }
    }
    __nv_bfloat16* op = out + row * ldo;
    *reinterpret_cast<uint4*>(op) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
    *reinterpret_cast<uint4*>(op + half) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
  }
}

}  // namespace hyc

using namespace hyc;

static int launch_rope(const RopeTensor& t0, const RopeTensor& t1, const void* cos_t, const void* sin_t, int64_t ld_table, int table_is_f32,
                       int64_t rows, int seq_len, int head_dim, int backward, void* stream) {
  const int64_t per_row = (int64_t)(t0.heads + t1.heads) * (head_dim / 16), bx = (per_row + 255) / 256;
  // one resident wave of blocks of 256 threads, each walking down the rows
  int64_t by = (int64_t)num_sms() * 8 / bx;
  by = by < 1 ? 1 : (by > rows ? rows : by);
  if (by > 65535) by = 65535;
  const dim3 grid((unsigned)bx, (unsigned)by);
  const float sgn = backward ? -1.f : 1.f;
  if (table_is_f32)
    launch_pdl(rope_kernel<true>, grid, dim3(256), 0, (cudaStream_t)stream, t0, t1, cos_t, sin_t, ld_table, rows, seq_len, head_dim, sgn);
  else
    launch_pdl(rope_kernel<false>, grid, dim3(256), 0, (cudaStream_t)stream, t0, t1, cos_t, sin_t, ld_table, rows, seq_len, head_dim, sgn);
  HYC_CHECK_LAUNCH();
  return HYC_OK;
}

extern "C" HYC_API int hyc_rope(const void* x, int64_t ldx, void* out, int64_t ldo, const void* cos_t, const void* sin_t,
                                int64_t ld_table, int table_is_f32, int64_t rows, int seq_len, int n_heads, int head_dim,
                                int backward, void* stream) {
  if (!x || !out || !cos_t || !sin_t) return HYC_ERR_NULL;
  if (rows < 0 || rows > 0xffffffffll || seq_len < 1 || n_heads < 1 || head_dim < 16 || (head_dim & 15) != 0) return HYC_ERR_SHAPE;
  if (ldx < (int64_t)n_heads * head_dim || ldo < (int64_t)n_heads * head_dim || ld_table < head_dim / 2) return HYC_ERR_SHAPE;
  if ((ldx & 7) != 0 || (ldo & 7) != 0 || (ld_table & (table_is_f32 ? 3 : 7)) != 0) return HYC_ERR_ALIGN;
  if (!aligned(x, 16) || !aligned(out, 16) || !aligned(cos_t, 16) || !aligned(sin_t, 16)) return HYC_ERR_ALIGN;
  if (rows == 0) return HYC_OK;
  return launch_rope({(const __nv_bfloat16*)x, (__nv_bfloat16*)out, ldx, ldo, n_heads}, {nullptr, nullptr, 0, 0, 0}, cos_t, sin_t, ld_table,
                     table_is_f32, rows, seq_len, head_dim, backward, stream);
}

extern "C" HYC_API int hyc_rope_pair(void* x0, int n_heads0, void* x1, int n_heads1, const void* cos_t, const void* sin_t, int64_t ld_table,
                                     int table_is_f32, int64_t rows, int seq_len, int head_dim, int backward, void* stream) {
  if (!x0 || !x1 || !cos_t || !sin_t) return HYC_ERR_NULL;
  if (rows < 0 || rows > 0xffffffffll || seq_len < 1 || n_heads0 < 1 || n_heads1 < 1 || head_dim < 16 || (head_dim & 15) != 0 ||
      ld_table < head_dim / 2) return HYC_ERR_SHAPE;
  if ((ld_table & (table_is_f32 ? 3 : 7)) != 0 || !aligned(x0, 16) || !aligned(x1, 16) || !aligned(cos_t, 16) || !aligned(sin_t, 16))
    return HYC_ERR_ALIGN;
  if (rows == 0) return HYC_OK;
  const int64_t ld0 = (int64_t)n_heads0 * head_dim, ld1 = (int64_t)n_heads1 * head_dim;
  return launch_rope({(const __nv_bfloat16*)x0, (__nv_bfloat16*)x0, ld0, ld0, n_heads0}, {(const __nv_bfloat16*)x1, (__nv_bfloat16*)x1, ld1, ld1, n_heads1},
                     cos_t, sin_t, ld_table, table_is_f32, rows, seq_len, head_dim, backward, stream);
}
