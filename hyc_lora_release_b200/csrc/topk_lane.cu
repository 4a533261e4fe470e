// Per-row top-k attention-map path, lane-per-group layout.
//
// A row of S = 64 * LPR columns (LPR = 1, 2, ..., 32 lanes per row) is spread over LPR adjacent lanes,
// every lane owning ONE quantization group: 64 consecutive columns = 128 contiguous bytes = 32 packed
// bf16 pairs.  A warp therefore works on 32 / LPR rows at a time, and everything that costs one warp
// instruction per row in a warp-per-row layout (reductions, scans, group parameters) is shared by
// those rows; group min/max needs no shuffle at all.  Rows whose groups are not a power of two (RAGGED) get the next power
// of two of lanes, of which the last ones own no group.
//
// Selection of the k largest magnitudes of a row is an exact radix select on BIT PLANES:
//   1. the lane's 64 magnitude patterns (15 bits) are bit-transposed in registers into 15 planes of
//      64 bits (plane b, bit c = bit b of the magnitude of the lane's column c): one byte-permute stage
//      and three shift/mask stages over 32 registers;
//   2. from the top plane down, one round per bit: ones = popc(plane & active) summed over the row's
//      lanes (one redux); if (count above + ones) >= k the bit of the threshold is 1 and the active set
//      shrinks to those elements, otherwise they are certainly selected ("greater" set) and leave the
//      active set.  Fifteen rounds of about a dozen instructions, whatever the data.
//   3. what is still active equals the threshold; those ties are taken in ascending column order.
// The selected elements are picked out of a shared-memory copy of the rows (which also zeroes them),
// staged as (column << 16 | value) words and written as one contiguous run per warp: the lists of
// adjacent rows are adjacent in memory.
#include "topk_lane.cuh"
#include "lane_group.cuh"

namespace hyc {

// sum over the LPR lanes of a row.  A whole warp uses the hardware reduction; for a part of a warp
// __reduce_add_sync with a partial mask is expanded into some twenty instructions, log2(LPR) butterfly
// steps are far cheaper (measured: 4.4 M of the kernel's 31 M warp instructions, 8 us of 47)
template <int LPR>
__device__ __forceinline__ int seg_add(int v) {
  if (LPR == 32) return (int)__reduce_add_sync(kFull, (unsigned)v);
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
template <int LPR>
__device__ __forceinline__ int seg_excl_scan(int v, int lr) {
  int incl = v;
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) {
    const int t = __shfl_up_sync(kFull, incl, o, LPR);
    if (lr >= o) incl += t;
  }
  return incl - v;
}

// w with only its n lowest set bits kept (n < popc(w))
__device__ __forceinline__ uint32_t keep_lowest_bits(uint32_t w, int n) {
  uint32_t r = w;
  for (int i = 0; i < n; ++i) r &= r - 1u;
  return w ^ r;
}

// A segment of LPR lanes serves one row, or (TWO) two rows: the first lanes one of them, the lanes behind the other.  The counts
// of both travel in one word, `shift` (0 or 16) says which half is the lane's own (a row has at most 2048 columns).
template <int LPR, bool TWO>
__device__ __forceinline__ int seg_total(int v, int shift) {
  if (!TWO) return seg_add<LPR>(v);
  return (seg_add<LPR>(v << shift) >> shift) & 0xffff;
}
template <int LPR, bool TWO>
__device__ __forceinline__ int seg_before(int v, int shift, int lr) {
  if (!TWO) return seg_excl_scan<LPR>(v, lr);
  return (seg_excl_scan<LPR>(v << shift, lr) >> shift) & 0xffff;
}

// The k entries of largest magnitude of the lane's row (see the top of this file), staged at `list` in column order and zeroed in
// the parked copy of the lane's group (sx).  col0: first column of that group; lanes that own no group or whose row is not
// valid select nothing.
template <int LPR, bool TWO>
__device__ __forceinline__ void select_top(const uint32_t (&xw)[32], uint32_t* sx, uint32_t* list, int k, bool owns, bool valid, int shift,
                                           uint32_t col0, int lr, int lane) {
        // ---- values paired (column c, column c + 16) so that the transposed planes come out in column
        // order: m[16 h + c] = (x[32 h + c], x[32 h + 16 + c]), c = 0..15.  Plane 15 (the signs) is never
        // read, so planes 14..0 are the magnitude patterns.
        uint32_t m[32];
  #pragma unroll
        for (int h = 0; h < 2; ++h)
  #pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t lo = xw[16 * h + i], hi = xw[16 * h + 8 + i];
            m[16 * h + 2 * i] = __byte_perm(lo, hi, 0x5410);
            m[16 * h + 2 * i + 1] = __byte_perm(lo, hi, 0x7632);
          }
        // ---- bit transpose.  Register index j = (h, c3 c2 c1 c0), bit position = (c4, b3 b2 b1 b0); every
        // stage swaps one index bit with one position bit, after the last one register 16 h + b holds
        // plane b of columns 32 h .. 32 h + 31 with column c at bit c.
  #pragma unroll
        for (int j = 0; j < 32; ++j)
          if ((j & 8) == 0) {
            const uint32_t x = m[j], y = m[j + 8];
            m[j] = __byte_perm(x, y, 0x6240);
            m[j + 8] = __byte_perm(x, y, 0x7351);
          }
  #pragma unroll
        for (int j = 0; j < 32; ++j)
          if ((j & 4) == 0) {
            const uint32_t x = m[j], y = m[j + 4];
            m[j] = (x & 0x0f0f0f0fu) | ((y << 4) & 0xf0f0f0f0u);
            m[j + 4] = ((x >> 4) & 0x0f0f0f0fu) | (y & 0xf0f0f0f0u);
          }
  #pragma unroll
        for (int j = 0; j < 32; ++j)
          if ((j & 2) == 0) {
            const uint32_t x = m[j], y = m[j + 2];
            m[j] = (x & 0x33333333u) | ((y << 2) & 0xccccccccu);
            m[j + 2] = ((x >> 2) & 0x33333333u) | (y & 0xccccccccu);
          }
  #pragma unroll
        for (int j = 0; j < 32; ++j)
          if ((j & 1) == 0) {
            const uint32_t x = m[j], y = m[j + 1];
            m[j] = (x & 0x55555555u) | ((y << 1) & 0xaaaaaaaau);
            m[j + 1] = ((x >> 1) & 0x55555555u) | (y & 0xaaaaaaaau);
          }
        // ---- radix select, most significant plane first
        // (branch-free: the rows of a warp take different sides)
        uint32_t A0 = owns ? kFull : 0u, A1 = A0, G0 = 0u, G1 = 0u;
        int rem = k;                       // k - (number of magnitudes known to be above the threshold)
  #pragma unroll
        for (int b = 14; b >= 0; --b) {
          const uint32_t x0 = m[b] & A0, x1 = m[16 + b] & A1;
          const int tot = seg_total<LPR, TWO>(__popc(x0) + __popc(x1), shift);
          const uint32_t drop = (tot >= rem) ? 0u : kFull;   // all ones: the threshold has a 0 here, the ones are above it
          G0 |= x0 & drop; G1 |= x1 & drop;
          A0 &= m[b] ^ drop; A1 &= m[16 + b] ^ drop;
          rem -= tot & (int)drop;
        }
        // ---- ties at the threshold: the first `rem` of them in column order
        {
          const int nt = __popc(A0) + __popc(A1);
          const int pre = seg_before<LPR, TWO>(nt, shift, lr);
          const int take = min(max(rem - pre, 0), nt);
          if (take < nt) {
            const int n0 = __popc(A0);
            if (take >= n0) { A1 = keep_lowest_bits(A1, take - n0); }
            else { A0 = keep_lowest_bits(A0, take); A1 = 0u; }
          }
        }
        uint32_t sel0 = G0 | A0, sel1 = G1 | A1;
        if (!valid) { sel0 = 0u; sel1 = 0u; }
        // ---- pick the selected elements (ascending columns) out of the parked copy and zero them there
        // (highest bit first, so the slots are filled from the lane's last one down)
        const int nsel = __popc(sel0) + __popc(sel1);
        uint32_t* slot = list + seg_before<LPR, TWO>(nsel, shift, lr) + nsel;
        uint16_t* sx16 = reinterpret_cast<uint16_t*>(sx);
        const uint32_t sw8 = (uint32_t)(lane & 7) << 3;          // chunk rotation, in halfword units
  #pragma unroll
        for (int h = 1; h >= 0; --h) {
          uint32_t bits = h ? sel1 : sel0;
          const uint32_t colh = (col0 + 32u * h) << 16;
          // two elements per trip: the busiest lane of the warp sets the number of trips (the large entries of a
          // causal row sit in few groups), and each trip is a load -> store chain
          while (bits) {
            const uint32_t e0 = 31u - (uint32_t)__clz(bits);
            bits ^= 1u << e0;
            const bool two = bits != 0u;
            const uint32_t e1 = two ? 31u - (uint32_t)__clz(bits) : e0;
            bits &= ~(1u << e1);
            uint16_t* at0 = sx16 + ((e0 + 32u * h) ^ sw8);
            uint16_t* at1 = sx16 + ((e1 + 32u * h) ^ sw8);
            const uint32_t v0 = *at0, v1 = *at1;
            *at0 = 0;
            *at1 = 0;                      // the same halfword again when there was only one
            slot[-1] = (colh + (e0 << 16)) | v0;
            if (two) slot[-2] = (colh + (e1 << 16)) | v1;
            slot -= two ? 2 : 1;
          }
        }
}

// The lists and codes of the warp's rows row0 .. row0 + n_rows - 1 (row: the lane's), whose groups are in xw and parked at sx
template <int QBIT, int LPR>
__device__ __forceinline__ void save_rows(uint32_t (&xw)[32], uint32_t* sx, uint32_t* so, int64_t row0, int n_rows, int64_t row, int GPR, int k,
                                          bool owns, bool valid, int lr, int rw, int lane, __nv_bfloat16* __restrict__ val_out,
                                          uint16_t* __restrict__ col_out, uint8_t* __restrict__ q, __nv_bfloat16* __restrict__ scale,
                                          int8_t* __restrict__ zp) {
  if (k > 0) {
    select_top<LPR, false>(xw, sx, so + rw * k, k, owns, valid, 0, 64u * (uint32_t)lr, lr, lane);
    __syncwarp();
    lane_slot_load(sx, lane, xw);
    // the lists of the warp's rows are one contiguous run
    const int n_ent = n_rows * k;
    __nv_bfloat16* vrun = val_out + row0 * k;
    uint16_t* crun = col_out + row0 * k;
    for (int j = lane; j < n_ent; j += 32) {
      const uint32_t w = so[j];
      vrun[j] = __ushort_as_bfloat16((uint16_t)(w & 0xffffu));
      crun[j] = (uint16_t)(w >> 16);
    }
  }
  float mn, mx;
  lane_minmax(xw, mn, mx);
  const GroupParams p = group_params<QBIT>(mn, mx);
  if (valid && owns) {
    lane_quant_store<QBIT>(xw, p, q + row * ((int64_t)GPR * (8 * QBIT)) + (64 * QBIT / 8) * lr);
    scale[row * GPR + lr] = __ushort_as_bfloat16(f32_to_bf16bits_rn(p.s));
    zp[row * GPR + lr] = (int8_t)(int)p.z;
  }
}

// What the SOFTMAX form of the compress kernel needs besides the map itself: the raw scores are read from `a`, turned
// into probabilities (scale, additive mask, softmax with the rounding points of softmax_fwd_kernel in
// norm_softmax.cu), written to `dense` for the P.V product, and saved in the same pass.
struct SoftmaxPrologue {
  float scale;
  const __nv_bfloat16* mask;     // additive mask or NULL; row m of (batch b, head h) at mask + b * mb + h * mh + m * S
  int64_t mb, mh;
  int heads, M;                  // rows = batch * heads * M, M a multiple of the rows a warp takes
  __nv_bfloat16* dense;          // [rows, S] probabilities (may be the scores buffer itself)
};

// ---------------------------------------------------------------- compress
template <int QBIT, int LPR, bool SOFTMAX, bool RAGGED>
__global__ void __launch_bounds__(256, HYC_LANE_MINB)
topk_lane_compress_kernel(const __nv_bfloat16* __restrict__ a, int64_t rows, int groups, int k,
                          __nv_bfloat16* __restrict__ val_out, uint16_t* __restrict__ col_out,
                          uint8_t* __restrict__ q, __nv_bfloat16* __restrict__ scale, int8_t* __restrict__ zp,
                          SoftmaxPrologue sp) {
  pdl_wait();
  constexpr int RPW = 32 / LPR;          // rows per warp
  const int GPR = RAGGED ? groups : LPR; // groups per row
  const int S = 64 * GPR;
  const LaneMap<LPR, RAGGED> map(GPR);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int lr = lane & (LPR - 1), rw = lane / LPR;
  const bool owns = !RAGGED || lr < GPR;
  __shared__ __align__(16) uint32_t s_x[8][32 * 32];          // the warp's rows, 128 bytes per lane
  __shared__ uint32_t s_out[8][kLaneStageEntries];            // staged (column << 16 | value) words
  uint32_t* sx = s_x[warp] + lane * 32;
  uint32_t* so = s_out[warp];
  const int64_t items = (rows + RPW - 1) / RPW;
  for (int64_t item = (int64_t)blockIdx.x * nwarps + warp; item < items; item += (int64_t)gridDim.x * nwarps) {
    const int64_t row0 = item * RPW, row = row0 + rw;
    const bool valid = row < rows;
    // the warp's rows are one contiguous run of 4 KB: fetch it, park it, read the lane's own group back
    const int64_t left = rows - row0;
    const int n_rows = (int)(left < RPW ? left : RPW);
    lane_run_to_shared(a + row0 * S, n_rows * (S / 16), s_x[warp], lane, map);
    __syncwarp();
    uint32_t xw[32];
    lane_slot_load(sx, lane, xw);

    if (SOFTMAX) {
      // ---- scores -> probabilities.  u = bf16(bf16(s * scale) + mask) replaces the raw scores in xw; the row maximum,
      // the exponentials and their sum are fp32; p = bf16(e / sum).  The exponentials are evaluated twice (once for
      // the sum, once for the result) instead of keeping 64 fp32 values per lane alive.
      constexpr float kLog2e = 1.4426950408889634f;
      __syncwarp();
      if (sp.mask != nullptr) {
        const int64_t bh = row0 / sp.M;
        const int m0 = (int)(row0 - bh * sp.M);
        lane_run_to_shared(sp.mask + (bh / sp.heads) * sp.mb + (bh % sp.heads) * sp.mh + (int64_t)m0 * S, n_rows * (S / 16),
                           s_x[warp], lane);
        __syncwarp();
      }
      __nv_bfloat162 hmx = __float2bfloat162_rn(-INFINITY);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4 mk = make_uint4(0u, 0u, 0u, 0u);
        if (sp.mask != nullptr) mk = *reinterpret_cast<const uint4*>(sx + park_chunk(c, lane));
        const uint32_t mw[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t t = pack_bf16x2_rn(bf16lo_to_f32(xw[4 * c + j]) * sp.scale, bf16hi_to_f32(xw[4 * c + j]) * sp.scale);
          if (sp.mask != nullptr)
            t = pack_bf16x2_rn(bf16lo_to_f32(t) + bf16lo_to_f32(mw[j]), bf16hi_to_f32(t) + bf16hi_to_f32(mw[j]));
          xw[4 * c + j] = t;
          hmx = __hmax2(hmx, *reinterpret_cast<const __nv_bfloat162*>(&t));
        }
      }
      float mx = fmaxf(__bfloat162float(hmx.x), __bfloat162float(hmx.y));
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
      const float mxl = mx * kLog2e;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        sum += exp2f(fmaf(bf16lo_to_f32(xw[j]), kLog2e, -mxl)) + exp2f(fmaf(bf16hi_to_f32(xw[j]), kLog2e, -mxl));
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) sum += __shfl_xor_sync(kFull, sum, o);
      const float inv = 1.0f / sum;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        xw[j] = pack_bf16x2_rn(exp2f(fmaf(bf16lo_to_f32(xw[j]), kLog2e, -mxl)) * inv,
                               exp2f(fmaf(bf16hi_to_f32(xw[j]), kLog2e, -mxl)) * inv);
      // the probabilities go to the parked copy (the emission below picks its entries there) and out as the dense map
      __syncwarp();
      lane_slot_store(sx, lane, xw);
      __syncwarp();
      lane_shared_to_run(s_x[warp], sp.dense + row0 * S, n_rows * (S / 16), lane);
      __syncwarp();
    }

    save_rows<QBIT, LPR>(xw, sx, so, row0, n_rows, row, GPR, k, owns, valid, lr, rw, lane, val_out, col_out, q, scale, zp);
    __syncwarp();   // the slots and the staging area are rewritten by other lanes in the next round
  }
}

// ---------------------------------------------------------------- compress, square maps whose rows end early
// Rows of a causal map have nothing behind their own position: half of the lanes of the kernel above work on zeros.  Here two
// rows share the LPR lanes of a segment where their groups fit side by side: rows of the last 128 stay alone, the 128-row
// tiles before them are paired outside in (the longest with the shortest), a tile left over in the middle with itself.
// Which rows fit is decided by their lengths; two that do not take the segment one after the other.  Groups behind a
// row's end are not read; they get the codes of a group of zeros.  What is stored is what the kernel above stores.
// That pays where rows end early: whole rows, taken two to a segment one after the other, make items twice as long and a last
// round half empty.  So the first row decides: where it is whole (no causal map), rows go one by one.  The shape of the launch
// is that of rows one by one, too: with the one that suits the pairs, five warps per block, fewer warps share an SM (31 % of them
// against 39 %).  us, 5 %, 4 bits, the kernel above / this one: causal [1,32,2048,2048] 142 / 104, [4,32,1024,1024]
// 154 / 116, [4,32,256,256] 12.0 / 11.6; nothing ruled out 130 / 126, 138 / 136, 11.7 / 12.0 (before the first row decided and with
// the other shape: 108, 126, 11.9; 160, 178, 17.1).
struct SquareMap { int M, items; };      // columns and rows of a map; segments of work per map
inline SquareMap square_map(int M) {
  const int full = (M - 1) / 128;
  return {M, M - 128 * full + 128 * (full / 2) + 64 * (full & 1)};
}
__device__ __forceinline__ void paired_rows(int i, int M, int& ra, int& rb) {
  const int full = (M - 1) / 128, last = M - 128 * full;
  if (i < last) { ra = 128 * full + i; rb = -1; return; }
  i -= last;
  const int p = i >> 7;
  if (p < full / 2) { ra = 128 * (full - 1 - p) + (i & 127); rb = 128 * p + (i & 127); return; }
  rb = 128 * p + (i & 127);
  ra = rb + 64;
}

template <int QBIT, int LPR, bool RAGGED>
__global__ void __launch_bounds__(256, HYC_LANE_MINB)
topk_lane_compress_cols_kernel(const __nv_bfloat16* __restrict__ a, int64_t rows, SquareMap sm, const uint16_t* __restrict__ row_cols, int k,
                               __nv_bfloat16* __restrict__ val_out, uint16_t* __restrict__ col_out,
                               uint8_t* __restrict__ q, __nv_bfloat16* __restrict__ scale, int8_t* __restrict__ zp) {
  pdl_wait();
  constexpr int RPW = 32 / LPR;
  constexpr uint32_t NONE = 0xffffffffu;
  const int GPR = sm.M / 64, kg = max((k + 63) / 64, 1);  // the k entries of a row lie in its groups and, if those are fewer, in the first kg
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int lr = lane & (LPR - 1), rw = lane / LPR;
  __shared__ __align__(16) uint32_t s_x[8][32 * 32];
  __shared__ uint32_t s_out[8][kLaneStageEntries];
  uint32_t* sx = s_x[warp] + lane * 32;
  uint32_t* so = s_out[warp] + 2 * rw * k;                 // the lists of the segment's two rows
  if ((int)__ldg(row_cols) >= sm.M) {
    // rows one by one, as in the kernel above but for the lanes behind their ends
    const LaneMap<LPR, RAGGED> map(GPR);
    const bool owns = !RAGGED || lr < GPR;
    const int64_t items = rows / RPW;                      // (M is a multiple of 64)
    for (int64_t item = (int64_t)blockIdx.x * nwarps + warp; item < items; item += (int64_t)gridDim.x * nwarps) {
      const int64_t row0 = item * RPW, row = row0 + rw;
      const bool inside = 64 * lr < (int)__ldg(row_cols + row);
      lane_run_to_shared(a + row0 * sm.M, RPW * GPR * 4, s_x[warp], lane, map);
      __syncwarp();
      uint32_t xw[32];
      lane_slot_load(sx, lane, xw);
      if (!inside) {                                        // whatever lies there
#pragma unroll
        for (int j = 0; j < 32; ++j) xw[j] = 0u;
        lane_slot_store(sx, lane, xw);
      }
      save_rows<QBIT, LPR>(xw, sx, s_out[warp], row0, RPW, row, GPR, k, owns, true, lr, rw, lane, val_out, col_out, q, scale, zp);
      __syncwarp();
    }
    return;
  }
  const GroupParams zero = group_params<QBIT>(0.f, 0.f);
  const uint32_t zero_scale = f32_to_bf16bits_rn(zero.s);
  // a byte of codes of zeros, four times
  const uint32_t zc = (group_code_bits<QBIT>(0.f, zero) & ((1u << QBIT) - 1u)) * (QBIT == 8 ? 1u : (QBIT == 4 ? 0x11u : 0x55u)) * 0x01010101u;
  const uint32_t n_items = (uint32_t)(rows / sm.M) * (uint32_t)sm.items;
  for (uint32_t item = blockIdx.x * nwarps + warp; item * RPW < n_items; item += gridDim.x * nwarps) {
    const uint32_t seg = item * RPW + rw;
    const bool valid = seg < n_items;
    uint32_t rowa = 0u, rowb = NONE;
    // groups the row takes up here, groups it has in memory (its lanes write a row of GPR groups: a row_cols above M must not count)
    int ga = 0, gb = 0, la = 0, lb = 0;
    if (valid) {
      const uint32_t map = seg / (uint32_t)sm.items;
      int ra, rb;
      paired_rows((int)(seg - map * (uint32_t)sm.items), sm.M, ra, rb);
      rowa = map * (uint32_t)sm.M + (uint32_t)ra;
      la = min((int)__ldg(row_cols + rowa) / 64, GPR);
      ga = max(la, kg);
      if (rb >= 0) {
        rowb = map * (uint32_t)sm.M + (uint32_t)rb;
        lb = min((int)__ldg(row_cols + rowb) / 64, GPR);
        gb = max(lb, kg);
      }
    }
    const bool together = ga + gb <= LPR;                   // (one row alone always fits)
    const int rounds = __any_sync(kFull, !together) ? 2 : 1;
    for (int round = 0; round < rounds; ++round) {
      // the lane's row and group in this round
      const int na = round == 0 ? ga : 0, nb = together ? (round == 0 ? gb : 0) : (round == 0 ? 0 : gb);
      const bool second = lr >= na, owns = lr < na + nb;
      const int g = second ? lr - na : lr;
      const uint32_t row = second ? rowb : rowa;
      const uint32_t group = row * (uint32_t)GPR + (uint32_t)g;
      const uint32_t from = owns && g < (second ? lb : la) ? group : NONE;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int p = 32 * i + lane, owner = p >> 2, c0 = 2 * (p & 3);
        const uint32_t f = __shfl_sync(kFull, from, owner);
        uint32_t t[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        if (f != NONE) ld_stream_v8(a + (int64_t)f * 64 + 16 * (p & 3), t);
        uint32_t* dst = s_x[warp] + owner * 32;
        *reinterpret_cast<uint4*>(dst + park_chunk(c0, owner)) = make_uint4(t[0], t[1], t[2], t[3]);
        *reinterpret_cast<uint4*>(dst + park_chunk(c0 + 1, owner)) = make_uint4(t[4], t[5], t[6], t[7]);
      }
      __syncwarp();
      uint32_t xw[32];
      lane_slot_load(sx, lane, xw);
      if (k > 0) {
        select_top<LPR, true>(xw, sx, so + (second ? k : 0), k, owns, true, second ? 16 : 0, 64u * (uint32_t)g, lr, lane);
        __syncwarp();
        lane_slot_load(sx, lane, xw);
#pragma unroll
        for (int w = 0; w < 2; ++w)
          if ((w ? nb : na) > 0) {
            const int64_t at = (int64_t)(w ? rowb : rowa) * k;
            for (int j = lr; j < k; j += LPR) {
              const uint32_t v = so[w * k + j];
              val_out[at + j] = __ushort_as_bfloat16((uint16_t)(v & 0xffffu));
              col_out[at + j] = (uint16_t)(v >> 16);
            }
          }
      }
      float mn, mx;
      lane_minmax(xw, mn, mx);
      const GroupParams p = group_params<QBIT>(mn, mx);
      if (owns) {
        lane_quant_store<QBIT>(xw, p, q + (int64_t)group * (64 * QBIT / 8));
        scale[group] = __ushort_as_bfloat16(f32_to_bf16bits_rn(p.s));
        zp[group] = (int8_t)(int)p.z;
      }
      // groups behind the rows' ends
#pragma unroll
      for (int w = 0; w < 2; ++w)
        if ((w ? nb : na) > 0)
          for (int gz = (w ? nb : na) + lr; gz < GPR; gz += LPR) {
            const uint32_t gi = (w ? rowb : rowa) * (uint32_t)GPR + (uint32_t)gz;
#pragma unroll
            for (int i = 0; i < QBIT / 2; ++i) st_stream_v4(q + (int64_t)gi * (64 * QBIT / 8) + 16 * i, make_uint4(zc, zc, zc, zc));
            scale[gi] = __ushort_as_bfloat16((uint16_t)zero_scale);
            zp[gi] = (int8_t)(int)zero.z;
          }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------- restore
// SMBWD: instead of the restored map y itself, write the softmax backward of it for the upstream gradient
// `grad`:  out = (g - sum_row(bf16(y * g))) * y  (operators/softmax_kernels.py:7-38: the product is a bf16
// operation, the row sum and the rest fp32).  The restored map never goes to HBM.
// COLS: row r is needed up to column row_cols[r] only (a multiple of 64)
template <int QBIT, int LPR, bool SMBWD, bool RAGGED, bool COLS>
__global__ void __launch_bounds__(256, SMBWD ? 3 : HYC_LANE_MINB)      // SMBWD: two tiles per warp, 3 blocks fill the SM
topk_lane_restore_kernel(const __nv_bfloat16* __restrict__ val, const uint16_t* __restrict__ colv, int k, float inv_k,
                         const uint8_t* __restrict__ q, const __nv_bfloat16* __restrict__ scale,
                         const int8_t* __restrict__ zp, int64_t rows, int groups, const __nv_bfloat16* __restrict__ grad,
                         float oscale, __nv_bfloat16* __restrict__ ao, const uint16_t* __restrict__ row_cols) {
  pdl_wait();
  constexpr int RPW = 32 / LPR;
  const int GPR = RAGGED ? groups : LPR;
  const int S = 64 * GPR;
  const int64_t QLD = (int64_t)S * QBIT / 8;
  const LaneMap<LPR, RAGGED> map(GPR);
  constexpr int PRE = 4;                 // list entries per lane fetched before the de-quantization
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int lr = lane & (LPR - 1), rw = lane / LPR;
  const bool owns = !RAGGED || lr < GPR;
  // dynamic shared memory: per warp its rows (128 bytes per lane) and, SMBWD, a second tile for the gradient rows
  extern __shared__ __align__(16) uint32_t s_dyn[];
  uint32_t* s_xw = s_dyn + warp * 1024;
  uint32_t* s_gw = s_dyn + (nwarps + warp) * 1024;
  uint32_t* sx = s_xw + lane * 32;
  uint16_t* sw16 = reinterpret_cast<uint16_t*>(s_xw);
  const int64_t items = (rows + RPW - 1) / RPW;
  for (int64_t item = (int64_t)blockIdx.x * nwarps + warp; item < items; item += (int64_t)gridDim.x * nwarps) {
    const int64_t row0 = item * RPW, row = row0 + rw;
    const bool valid = row < rows;
    const int64_t left = rows - row0;
    const int n_rows = (int)(left < RPW ? left : RPW);
    const int n_ent = n_rows * k;
    bool wanted = valid && owns;
    if (COLS) wanted = wanted && lr < (int)__ldg(row_cols + row) / 64;
    // the gradient rows start their way into shared memory now and arrive while the map is being rebuilt
    if (SMBWD) lane_run_to_shared_async(grad + row0 * S, n_rows * (S / 16), s_gw, lane, map);
    const __nv_bfloat16* vrun = val + row0 * k;
    const uint16_t* crun = colv + row0 * k;
    uint16_t pc[PRE], pv[PRE];
#pragma unroll
    for (int i = 0; i < PRE; ++i) {
      const int j = lane + 32 * i;
      pc[i] = 0; pv[i] = 0;
      if (j < n_ent) { pc[i] = crun[j]; pv[i] = __bfloat16_as_ushort(vrun[j]); }
    }
    // de-quantize the lane's group into its shared-memory slot
    {
      uint32_t o[32];
      if (wanted) {
        const float s = __bfloat162float(scale[row * GPR + lr]);
        const float z = (float)zp[row * GPR + lr];
        lane_load_dequant<QBIT>(q + row * QLD + (64 * QBIT / 8) * lr, s, z, o);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = 0u;
      }
      lane_slot_store(sx, lane, o);
    }
    __syncwarp();
    // the outlier lists overwrite their entries there.  Entry j of the run belongs to row j / k of the warp:
    // (j + 0.5) / k is never within 1/(2k) of an integer, so the fp32 product truncates to the exact quotient.
    // Column c of that row lives in lane (row * LPR + c / 64), halfword (c % 64) rotated like the chunks.
#pragma unroll
    for (int i = 0; i < PRE; ++i) {
      const int j = lane + 32 * i;
      if (j < n_ent) {
        const int r = (int)(((float)j + 0.5f) * inv_k);
        const int owner = r * LPR + (pc[i] >> 6);
        sw16[owner * 64 + ((pc[i] & 63) ^ ((owner & 7) << 3))] = pv[i];
      }
    }
    for (int j = lane + 32 * PRE; j < n_ent; j += 32) {
      const int r = (int)(((float)j + 0.5f) * inv_k);
      const int c = crun[j];
      const int owner = r * LPR + (c >> 6);
      sw16[owner * 64 + ((c & 63) ^ ((owner & 7) << 3))] = __bfloat16_as_ushort(vrun[j]);
    }
    __syncwarp();
    if (SMBWD) {
      uint32_t yv[32], gv[32];
      lane_slot_load(sx, lane, yv);                       // the lane's own group of the restored row
      lane_async_wait();
      __syncwarp();
      lane_slot_load(s_gw + lane * 32, lane, gv);
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const __nv_bfloat162 p = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&yv[j]),
                                            *reinterpret_cast<const __nv_bfloat162*>(&gv[j]));
        acc += __bfloat162float(p.x) + __bfloat162float(p.y);
      }
      if (!owns) acc = 0.f;
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) acc += __shfl_xor_sync(kFull, acc, o);     // stays inside the row's lanes
#pragma unroll
      for (int j = 0; j < 32; ++j)
        gv[j] = pack_bf16x2_rn((bf16lo_to_f32(gv[j]) - acc) * bf16lo_to_f32(yv[j]),
                               (bf16hi_to_f32(gv[j]) - acc) * bf16hi_to_f32(yv[j]));
      if (oscale != 1.f) {        // a second bf16 operation on the result (the layer's `grad_s / sqrt(d)`)
#pragma unroll
        for (int j = 0; j < 32; ++j) gv[j] = pack_bf16x2_rn(bf16lo_to_f32(gv[j]) * oscale, bf16hi_to_f32(gv[j]) * oscale);
      }
      __syncwarp();
      lane_slot_store(sx, lane, gv);
      __syncwarp();
    }
    // the warp's rows leave as four fully coalesced 1 KB stores
    lane_shared_to_run(s_xw, ao + row0 * S, n_rows * (S / 16), lane, map, COLS ? __ballot_sync(kFull, wanted) : kFull);
    __syncwarp();
  }
}

// ---------------------------------------------------------------- softmax backward on dense maps
// out = (g - sum_row(bf16(y * g))) * y, same layout and staging as above
template <int LPR, bool RAGGED>
__global__ void __launch_bounds__(256, 3)
softmax_bwd_lane_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ g, int64_t rows, int groups,
                        float oscale, __nv_bfloat16* __restrict__ out) {
  pdl_wait();
  constexpr int RPW = 32 / LPR;
  const int GPR = RAGGED ? groups : LPR;
  const int S = 64 * GPR;
  const LaneMap<LPR, RAGGED> map(GPR);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  // dynamic shared memory: two 4 KB tiles per warp, so that both operands are on their way at once (cp.async)
  extern __shared__ __align__(16) uint32_t s_dyn[];
  uint32_t* s_yw = s_dyn + warp * 1024;
  uint32_t* s_gw = s_dyn + (nwarps + warp) * 1024;
  uint32_t* sx = s_yw + lane * 32;
  const int64_t items = (rows + RPW - 1) / RPW;
  for (int64_t item = (int64_t)blockIdx.x * nwarps + warp; item < items; item += (int64_t)gridDim.x * nwarps) {
    const int64_t row0 = item * RPW, left = rows - row0;
    const int n_pieces = (int)(left < RPW ? left : RPW) * (S / 16);
    uint32_t yv[32], gv[32];
    lane_run_to_shared_async(y + row0 * S, n_pieces, s_yw, lane, map);
    lane_run_to_shared_async(g + row0 * S, n_pieces, s_gw, lane, map);
    lane_async_wait();
    __syncwarp();
    lane_slot_load(sx, lane, yv);
    lane_slot_load(s_gw + lane * 32, lane, gv);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const __nv_bfloat162 p = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&yv[j]),
                                          *reinterpret_cast<const __nv_bfloat162*>(&gv[j]));
      acc += __bfloat162float(p.x) + __bfloat162float(p.y);
    }
    if (RAGGED && (lane & (LPR - 1)) >= GPR) acc = 0.f;
#pragma unroll
    for (int o = 1; o < LPR; o <<= 1) acc += __shfl_xor_sync(kFull, acc, o);
#pragma unroll
    for (int j = 0; j < 32; ++j)
      gv[j] = pack_bf16x2_rn((bf16lo_to_f32(gv[j]) - acc) * bf16lo_to_f32(yv[j]),
                             (bf16hi_to_f32(gv[j]) - acc) * bf16hi_to_f32(yv[j]));
    if (oscale != 1.f) {
#pragma unroll
      for (int j = 0; j < 32; ++j) gv[j] = pack_bf16x2_rn(bf16lo_to_f32(gv[j]) * oscale, bf16hi_to_f32(gv[j]) * oscale);
    }
    __syncwarp();
    lane_slot_store(sx, lane, gv);
    __syncwarp();
    lane_shared_to_run(s_yw, out + row0 * S, n_pieces, lane, map);
    __syncwarp();
  }
}

template <int LPR, bool RAGGED>
static void launch_softmax_bwd(const void* y, const void* g, int64_t rows, int groups, float oscale, void* out, cudaStream_t st) {
  auto kern = softmax_bwd_lane_kernel<LPR, RAGGED>;
  static bool attr[64] = {false};      // up to 64 KB of dynamic shared memory per block: set per device
  const int slot = current_device_slot();
  if (slot < 0 || !attr[slot]) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 8192);
    if (slot >= 0) attr[slot] = true;
  }
  int grid, threads;
  lane_launch_shape(kern, rows, 32 / LPR, grid, threads, 8192);
  launch_pdl(kern, dim3((unsigned)grid), dim3(threads), (threads / 32) * 8192, st, (const __nv_bfloat16*)y, (const __nv_bfloat16*)g, rows, groups, oscale,
                                                     (__nv_bfloat16*)out);
}

#define HYC_LANE_DISPATCH(FN, ...)                                                                    \
  switch (topk_lanes_per_row(S)) {                                                                    \
    case 1: FN(1, false)(__VA_ARGS__); break;                                                         \
    case 2: FN(2, false)(__VA_ARGS__); break;                                                         \
    case 4: if (S == 256) FN(4, false)(__VA_ARGS__); else FN(4, true)(__VA_ARGS__); break;            \
    case 8: if (S == 512) FN(8, false)(__VA_ARGS__); else FN(8, true)(__VA_ARGS__); break;            \
    case 16: if (S == 1024) FN(16, false)(__VA_ARGS__); else FN(16, true)(__VA_ARGS__); break;        \
    default: if (S == 2048) FN(32, false)(__VA_ARGS__); else FN(32, true)(__VA_ARGS__); break;        \
  }

// rows of 64 n <= 2048 columns, 32-byte aligned tensors; false = not covered (nothing launched)
bool softmax_bwd_lane(const void* y, const void* g, int64_t rows, int S, float oscale, void* out, cudaStream_t st) {
  if (S < 64 || S > 2048 || S % 64 != 0 || !aligned(y, 32) || !aligned(g, 32) || !aligned(out, 32)) return false;
#define FN(L, RG) launch_softmax_bwd<L, RG>
  HYC_LANE_DISPATCH(FN, y, g, rows, S / 64, oscale, out, st);
#undef FN
  return true;
}

// ---------------------------------------------------------------- launchers
template <int QBIT, int LPR, bool RAGGED>
static void launch_compress(const void* a, int64_t rows, int groups, int k, void* val, uint16_t* col, void* q, void* scale,
                            int8_t* zp, const SoftmaxPrologue* sp, cudaStream_t st) {
  int grid, threads;
  if (sp == nullptr) {
    auto kern = topk_lane_compress_kernel<QBIT, LPR, false, RAGGED>;
    lane_launch_shape(kern, rows, 32 / LPR, grid, threads);
    launch_pdl(kern, dim3((unsigned)grid), dim3(threads), 0, st, (const __nv_bfloat16*)a, rows, groups, k, (__nv_bfloat16*)val, col,
                                   (uint8_t*)q, (__nv_bfloat16*)scale, zp, SoftmaxPrologue{});
  } else if constexpr (!RAGGED) {
    auto kern = topk_lane_compress_kernel<QBIT, LPR, true, false>;
    lane_launch_shape(kern, rows, 32 / LPR, grid, threads);
    launch_pdl(kern, dim3((unsigned)grid), dim3(threads), 0, st, (const __nv_bfloat16*)a, rows, groups, k, (__nv_bfloat16*)val, col,
                                   (uint8_t*)q, (__nv_bfloat16*)scale, zp, *sp);
  }
}
template <int QBIT, int LPR, bool RAGGED>
static void launch_compress_cols(const void* a, int64_t rows, int M, const uint16_t* row_cols, int k, void* val, uint16_t* col, void* q, void* scale,
                                 int8_t* zp, cudaStream_t st) {
  const SquareMap sm = square_map(M);
  auto kern = topk_lane_compress_cols_kernel<QBIT, LPR, RAGGED>;
  int grid, threads;
  lane_launch_shape(kern, rows, 32 / LPR, grid, threads);
  launch_pdl(kern, dim3((unsigned)grid), dim3(threads), 0, st, (const __nv_bfloat16*)a, rows, sm, row_cols, k, (__nv_bfloat16*)val, col,
             (uint8_t*)q, (__nv_bfloat16*)scale, zp);
}
template <int QBIT, int LPR, bool RAGGED>
static void launch_restore(const void* val, const uint16_t* col, int k, const void* q, const void* scale, const int8_t* zp, int64_t rows, int groups,
                           const uint16_t* row_cols, const void* grad, float oscale, void* ao, cudaStream_t st) {
  auto run = [&](auto kern, int bytes_per_warp) {
    int grid, threads;
    lane_launch_shape(kern, rows, 32 / LPR, grid, threads, bytes_per_warp);
    launch_pdl(kern, dim3((unsigned)grid), dim3(threads), (threads / 32) * bytes_per_warp, st, (const __nv_bfloat16*)val, col, k,
               k > 0 ? 1.0f / (float)k : 0.f, (const uint8_t*)q, (const __nv_bfloat16*)scale, zp, rows, groups, (const __nv_bfloat16*)grad, oscale,
               (__nv_bfloat16*)ao, row_cols);
  };
  if (row_cols != nullptr) {
    run(topk_lane_restore_kernel<QBIT, LPR, false, RAGGED, true>, 4096);
  } else if (grad == nullptr) {
    run(topk_lane_restore_kernel<QBIT, LPR, false, RAGGED, false>, 4096);
  } else {
    auto kern = topk_lane_restore_kernel<QBIT, LPR, true, RAGGED, false>;
    // two 4 KB tiles per warp: up to 64 KB per block, above the default limit (set per device)
    static bool attr[64] = {false};
    const int slot = current_device_slot();
    if (slot < 0 || !attr[slot]) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 8192);
      if (slot >= 0) attr[slot] = true;
    }
    run(kern, 8192);
  }
}

template <int QB>
static int compress_q(const void* a, int64_t rows, int S, int k, void* val, uint16_t* col, void* q, void* scale,
                      int8_t* zp, const SoftmaxPrologue* sp, cudaStream_t st) {
#define FN(L, RG) launch_compress<QB, L, RG>
  HYC_LANE_DISPATCH(FN, a, rows, S / 64, k, val, col, q, scale, zp, sp, st);
#undef FN
  return HYC_OK;
}
template <int QB>
static int restore_q(const void* val, const uint16_t* col, int k, const void* q, const void* scale, const int8_t* zp,
                     int64_t rows, int S, const uint16_t* row_cols, const void* grad, float oscale, void* ao, cudaStream_t st) {
#define FN(L, RG) launch_restore<QB, L, RG>
  HYC_LANE_DISPATCH(FN, val, col, k, q, scale, zp, rows, S / 64, row_cols, grad, oscale, ao, st);
#undef FN
  return HYC_OK;
}

int topk_lane_compress(const void* a, int64_t rows, int S, int k, void* val_out, uint16_t* col_out,
                       void* q_out, void* scale_out, int8_t* zp_out, int q_bit, cudaStream_t st) {
  if (!topk_lane_ok(S, k)) return HYC_ERR_SHAPE;
  if (q_bit == 2) return compress_q<2>(a, rows, S, k, val_out, col_out, q_out, scale_out, zp_out, nullptr, st);
  if (q_bit == 4) return compress_q<4>(a, rows, S, k, val_out, col_out, q_out, scale_out, zp_out, nullptr, st);
  return compress_q<8>(a, rows, S, k, val_out, col_out, q_out, scale_out, zp_out, nullptr, st);
}

// scores [rows, S] -> probabilities (written to `dense`) and their saved form, one pass.  Covered: the shapes of
// topk_lane_ok with S a power of two, M a multiple of the rows a warp takes and mask rows S apart; HYC_ERR_UNSUPPORTED otherwise
// (nothing launched: the caller runs the softmax and the compress kernels one after the other).
int topk_lane_softmax_compress(const void* scores, float sc, const void* mask, int64_t mb, int64_t mh, int64_t mr, int heads,
                               int M, int64_t rows, int S, int k, void* dense, void* val_out, uint16_t* col_out,
                               void* q_out, void* scale_out, int8_t* zp_out, int q_bit, cudaStream_t st) {
  if (!topk_lane_ok(S, k) || (S & (S - 1)) != 0) return HYC_ERR_UNSUPPORTED;
  const int rpw = 32 / (S / 64);
  if (M % rpw != 0 || (mask != nullptr && mr != S) || !aligned(scores, 32) || !aligned(dense, 32) || !aligned(q_out, 32) ||
      (mask != nullptr && (!aligned(mask, 32) || (mb & 15) != 0 || (mh & 15) != 0)))
    return HYC_ERR_UNSUPPORTED;
  SoftmaxPrologue sp;
  sp.scale = sc; sp.mask = (const __nv_bfloat16*)mask; sp.mb = mb; sp.mh = mh; sp.heads = heads; sp.M = M;
  sp.dense = (__nv_bfloat16*)dense;
  if (q_bit == 2) return compress_q<2>(scores, rows, S, k, val_out, col_out, q_out, scale_out, zp_out, &sp, st);
  if (q_bit == 4) return compress_q<4>(scores, rows, S, k, val_out, col_out, q_out, scale_out, zp_out, &sp, st);
  return compress_q<8>(scores, rows, S, k, val_out, col_out, q_out, scale_out, zp_out, &sp, st);
}
int topk_lane_restore(const void* val, const uint16_t* col, int k, const void* q, const void* scale,
                      const int8_t* zp, int64_t rows, int S, const uint16_t* row_cols, const void* grad_or_null, float out_scale, void* a_out,
                      int q_bit, cudaStream_t st) {
  if (!topk_lane_ok(S, k)) return HYC_ERR_SHAPE;
  if (q_bit == 2) return restore_q<2>(val, col, k, q, scale, zp, rows, S, row_cols, grad_or_null, out_scale, a_out, st);
  if (q_bit == 4) return restore_q<4>(val, col, k, q, scale, zp, rows, S, row_cols, grad_or_null, out_scale, a_out, st);
  return restore_q<8>(val, col, k, q, scale, zp, rows, S, row_cols, grad_or_null, out_scale, a_out, st);
}

template <int QB>
static int compress_cols_q(const void* a, int64_t rows, int M, const uint16_t* row_cols, int k, void* val, uint16_t* col, void* q, void* scale,
                           int8_t* zp, cudaStream_t st) {
  const int S = M;
#define FN(L, RG) launch_compress_cols<QB, L, RG>
  HYC_LANE_DISPATCH(FN, a, rows, M, row_cols, k, val, col, q, scale, zp, st);
#undef FN
  return HYC_OK;
}
int topk_lane_compress_cols(const void* a, int64_t rows, int M, const uint16_t* row_cols, int k, void* val_out, uint16_t* col_out,
                            void* q_out, void* scale_out, int8_t* zp_out, int q_bit, cudaStream_t st) {
  if (!topk_lane_cols_ok(M, k)) return HYC_ERR_UNSUPPORTED;
  if (q_bit == 2) return compress_cols_q<2>(a, rows, M, row_cols, k, val_out, col_out, q_out, scale_out, zp_out, st);
  if (q_bit == 4) return compress_cols_q<4>(a, rows, M, row_cols, k, val_out, col_out, q_out, scale_out, zp_out, st);
  return compress_cols_q<8>(a, rows, M, row_cols, k, val_out, col_out, q_out, scale_out, zp_out, st);
}

}  // namespace hyc
