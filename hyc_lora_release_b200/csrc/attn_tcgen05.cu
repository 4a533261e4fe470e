// Attention of the fused layer on tcgen05: softmax(Q K^T * scale + mask) V in one kernel and its backward pass in two,
// for heads of 128 columns.  Operands stay in the hidden layout [B, M, heads * 128] (three-dimensional tensor maps cut
// a head's 128-row tile out of it, rows past the sequence read as zero), grouped key/value heads are addressed, not
// copied.
//
//   forward   a CTA owns 128 query rows of one head and walks the key tiles twice: first for the row maxima and sums,
//             then for the probabilities (rounded to bf16 exactly where the separate kernels round) and P V.  The
//             scores never leave tensor memory; recomputing them costs one more product per tile, a round trip through
//             HBM cost four passes over the [B, heads, M, M] map.
//   backward  q kernel: per 128 query rows dP = dO V^T tile by tile, first for D = rowsum(P * dP) on the restored map,
//             then for dS = (dP - D) * P * scale and dQ += dS K; dS goes to HBM once.
//             kv kernel: per 128 keys dV += P^T dO and dK += dS^T Q over the query tiles and the heads of the group.
//
// Tiles that the additive mask rules out completely (a causal map: nearly half) are skipped everywhere; a small kernel
// classifies the mask's tiles on every call.  In the map they are written as zeros, or, where the caller takes the ends of the
// rows (row_cols), only those in front of a tile that is not ruled out.
//
// CTA (one per SM): warp 0 loads (TMA, ring of 32 KB tiles), warp 1 issues the MMAs, the other sixteen (kv kernel: eight)
// do the element-wise work, each a 32-row quadrant and a quarter of the tile's columns (with eight warps of 64 columns
// the schedulers issued 0.3 instructions a cycle; [1,32,2048,2048] forward, in an earlier state, 173 us against 139 us with sixteen).  Scores /
// dP are double-buffered in tensor memory, so the next tile's product runs while this one is worked on; P and dS go back
// to tensor memory as the A operand of the second product.  Every wait is bounded (see tc_common.cuh).
//
// What bounds them: the forward and q kernels the element-wise work (issue slots 0.46 and 0.36 of one per cycle and
// scheduler, waits on tensor memory and loads in between; DRAM at 21 and 49 %), the kv kernel its loads (two 32 KB tiles per
// product; issue slots 0.07, DRAM 59 %).  The tensor pipe is busy a quarter of the time in all three.  Measured
// [1,32,2048,2048] causal, cold: forward 106 us with the ends of the rows and 122 with the whole map, for 512 MB of map traffic saved;
// backward 105.5 + 65.2 as single launches (the two between a pair of events: 179); the separate steps took 110 + 104 + 107 us (products, softmax) and 330 us.
#include "tc_common.cuh"
#include <math.h>

namespace hyc {
namespace at {

using namespace tc;

constexpr int TILE = 128, TILE_BYTES = TILE * TILE * 2;
constexpr int EW = 16;                           // element-wise warps of the forward and q kernels
constexpr int KV_WARPS = 8;                      // of the kv kernel
constexpr int AT_THREADS = 64 + 32 * EW, KV_THREADS = 64 + 32 * KV_WARPS;
constexpr int MAX_TILES = 32;                    // sequence lengths up to 4096

// one entry per 128 x 128 tile of the mask: 0 all zero, 1 mixed, 2 nothing passes; rows: bit set = the row has an entry
// that passes in this tile
struct __align__(16) TileClass { uint32_t rows[4]; uint32_t cls; uint32_t pad[3]; };
constexpr float kMaskedOut = -1e30f;             // at or below: exp of the masked score is zero next to any that passes

struct AttnParams {
  int B, M, heads, kv_heads, tiles;
  float scale;
  const __nv_bfloat16* mask;                     // additive [b or 1, h or 1, M, M], or null
  int64_t mb, mh, mr;
  const TileClass* cls;                          // [b or 1][h or 1][tiles][tiles], or null (no tile is skipped)
  int64_t cls_b, cls_h;
  __nv_bfloat16* out0;                           // forward: o; q kernel: grad_q; kv kernel: grad_k
  __nv_bfloat16* out1;                           // kv kernel: grad_v
  __nv_bfloat16* map;                            // forward: probabilities [B * heads, M, M]; q kernel: dS
  const __nv_bfloat16* code_scale;               // forward: per-channel scale of o, or null
  uint8_t* codes;                                // forward: packed codes of o
  uint16_t* row_cols;                            // forward: columns of each map row from which on nothing is written, or null
  int* status;
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// a 128 x 128 tile as two boxes of 64 columns
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int col, int row, int z) {
  mbar_expect_tx(bar, TILE_BYTES);
  tma_load_3d(dst, map, smem_u32(bar), col, row, z);
  tma_load_3d(dst + TILE_BYTES / 2, map, smem_u32(bar), col + 64, row, z);
}
// operand descriptors of a tile for K step kk (16 of 128): rows x K (K contiguous), or K x columns (K = tile rows)
__device__ __forceinline__ uint64_t desc_k(uint32_t tile, int kk) {
  return make_desc(tile + (uint32_t)((kk >> 2) * (TILE_BYTES / 2) + (kk & 3) * 32), 16, 1024);
}
__device__ __forceinline__ uint64_t desc_mn(uint32_t tile, int kk) { return make_desc(tile + (uint32_t)(kk * 2048), TILE_BYTES / 2, 1024); }
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TILE >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
constexpr uint32_t kAMn = 1u << 15, kBMn = 1u << 16;

// A operand from tensor memory (bf16 pairs, one K step = 8 columns)
__device__ __forceinline__ void tc_mma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
      ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// two fp32 lanes per instruction; the lanes round like the scalar operations
__device__ __forceinline__ float2 mul2f(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2f(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2f(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 unpack2(uint32_t v) { return make_float2(bf16lo_to_f32(v), bf16hi_to_f32(v)); }
__device__ __forceinline__ uint32_t pack2(float2 v) { return pack_bf16x2_rn(v.x, v.y); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) { return as_u32(__hmax2(as_bf2(a), as_bf2(b))); }
constexpr float kLog2e = 1.4426950408889634f;
// exp(u - m) is evaluated as 2^(u * k - m * k).  Where m itself is a masked score m * log2(e) could overflow.  k = 1 does there:
// u and m are bf16 values, so they are equal (2^0) or at least 2^-8 of 1e30 apart (2^-inf = 0), whatever the base
__device__ __forceinline__ float exp_scale(float m) { return m <= kMaskedOut ? 1.f : kLog2e; }
constexpr uint32_t kNegInf2 = 0xff80ff80u;

// a warp's [32 rows][32 columns] tile to rows of `ld` elements, clipped to `cols` columns (a multiple of 8)
__device__ __forceinline__ void flush_clipped(const uint32_t* R, __nv_bfloat16* out, int row0, int rows, int64_t ld, int n, int cols, int lane) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = 8 * k + (lane >> 2), c = n + 8 * (lane & 3);
    const uint4 v = *reinterpret_cast<const uint4*>(R + gd_chunk(r, lane & 3));
    if (row0 + r < rows && c < cols) *reinterpret_cast<uint4*>(out + (int64_t)(row0 + r) * ld + c) = v;
  }
}
// 32 fp32 accumulator columns of the lane's row into the warp's tile as bf16
__device__ __forceinline__ void put_row_bf16(uint32_t* R, int lane, const uint32_t (&acc)[32]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = pack_bf16x2_rn(__uint_as_float(acc[8 * e + 2 * i]), __uint_as_float(acc[8 * e + 2 * i + 1]));
    *reinterpret_cast<uint4*>(R + gd_chunk(lane, e)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
__device__ __forceinline__ void at_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * EW) : "memory"); }

// ------------------------------------------------------------------ mask classes
__global__ void __launch_bounds__(256)
mask_class_kernel(const __nv_bfloat16* __restrict__ mask, int64_t mb, int64_t mh, int64_t mr, int M, int tiles, int mask_heads, TileClass* __restrict__ out) {
  pdl_wait();
  __shared__ uint32_t s_rows[4], s_nonzero;
  const int kt = blockIdx.x, qt = blockIdx.y, z = blockIdx.z;
  if (threadIdx.x < 4) s_rows[threadIdx.x] = 0u;
  if (threadIdx.x == 4) s_nonzero = 0u;
  __syncthreads();
  const __nv_bfloat16* base = mask + (z / mask_heads) * mb + (z % mask_heads) * mh;
  // 16 lanes x 8 columns per row, 16 rows per step; all of a thread's eight loads are on their way before the first use
  uint4 v[8];
  const int col = kt * TILE + 8 * (threadIdx.x & 15);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = qt * TILE + (threadIdx.x >> 4) + 16 * i;
    v[i] = make_uint4(0xff7fff7fu, 0xff7fff7fu, 0xff7fff7fu, 0xff7fff7fu);      // outside: nothing passes
    if (row < M && col < M) v[i] = *reinterpret_cast<const uint4*>(base + (int64_t)row * mr + col);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = (threadIdx.x >> 4) + 16 * i;
    const bool inside = qt * TILE + r < M && col < M;
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
    bool pass = false, nonzero = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      pass |= !(bf16lo_to_f32(w[e]) <= kMaskedOut) | !(bf16hi_to_f32(w[e]) <= kMaskedOut);
      nonzero |= inside && ((w[e] & 0x7fff7fffu) != 0u);
    }
    if (pass) atomicOr(&s_rows[r >> 5], 1u << (r & 31));
    if (nonzero) s_nonzero = 1u;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    TileClass t = {};
    uint32_t any = 0u;
    for (int i = 0; i < 4; ++i) { t.rows[i] = s_rows[i]; any |= s_rows[i]; }
    t.cls = any == 0u ? 2u : (s_nonzero ? 1u : 0u);
    out[((int64_t)z * tiles + qt) * tiles + kt] = t;
  }
}

// the class of tile (qt, kt); "ruled out" only if every row of the query tile has an entry that passes somewhere (a row
// that is masked everywhere has equal scores, not none)
__device__ __forceinline__ uint32_t class_of(const AttnParams& p, int b, int h, int qt, int kt) {
  if (p.cls == nullptr) return p.mask != nullptr ? 1u : 0u;
  const TileClass* t = p.cls + ((b * p.cls_b + h * p.cls_h) * p.tiles + qt) * p.tiles;
  uint32_t rows[4] = {0u, 0u, 0u, 0u};
  for (int i = 0; i < p.tiles; ++i) {
    const uint4 r = *reinterpret_cast<const uint4*>(t[i].rows);
    rows[0] |= r.x; rows[1] |= r.y; rows[2] |= r.z; rows[3] |= r.w;
  }
  bool rows_ok = true;
  const int left = p.M - qt * TILE;
  for (int i = 0; i < 4; ++i) {
    const int n = left - 32 * i;
    const uint32_t need = n >= 32 ? 0xffffffffu : (n > 0 ? (1u << n) - 1u : 0u);
    rows_ok = rows_ok && (rows[i] & need) == need;
  }
  const uint32_t c = t[kt].cls;
  return c == 2u && !rows_ok ? 1u : c;
}

// ------------------------------------------------------------------ shared-memory plan
//   forward:   the resident tile (Q), RING ring slots, a 2 KB tile per element-wise warp, row values
//   q kernel:  the resident tile (dO), Q_RING ring slots, row values
//   kv kernel: KV_SLOTS ring slots, eight 2 KB tiles
// then the barriers
constexpr int RING = 4, KV_SLOTS = 6;
constexpr int AT_EPI = TILE_BYTES * (1 + RING), KV_EPI = TILE_BYTES * KV_SLOTS;
constexpr int AT_ROWS = AT_EPI + EW * 2048;
constexpr int AT_BARS = AT_ROWS + 8 * TILE * 4, KV_BARS = KV_EPI + KV_WARPS * 2048;
constexpr int Q_RING = 6, Q_ROWS = TILE_BYTES * (1 + Q_RING), Q_BARS = Q_ROWS + 2 * TILE * 4;
constexpr int AT_SMEM = 1024 + AT_BARS + 512, KV_SMEM = 1024 + KV_BARS + 512, Q_SMEM = 1024 + Q_BARS + 512;
static_assert(Q_SMEM <= 227 * 1024 && AT_SMEM <= 227 * 1024 && KV_SMEM <= 227 * 1024, "shared memory of a block");
constexpr int MAX_SLOTS = 6;

struct Bars {
  uint64_t *full, *empty;        // [MAX_SLOTS]
  uint64_t *res_full;            // the resident tile
  uint64_t *s_full, *s_free;     // [2] a product is in its buffer / has been read (first pass)
  uint64_t *p_full;              // [2] the element-wise result is in tensor memory
  uint64_t* acc_full;            // accumulator complete
  uint64_t* ds_out;              // [2] q kernel: dS has left its slot
  uint32_t* tmem_slot;
  volatile int* abort_flag;
  uint8_t* cls;                  // [MAX_TILES]
  __device__ __forceinline__ explicit Bars(uint8_t* at) {
    uint64_t* b = reinterpret_cast<uint64_t*>(at);
    full = b; empty = b + MAX_SLOTS; res_full = b + 2 * MAX_SLOTS;
    s_full = res_full + 1; s_free = s_full + 2; p_full = s_free + 2; acc_full = p_full + 2;
    ds_out = acc_full + 1;
    tmem_slot = reinterpret_cast<uint32_t*>(ds_out + 2);
    abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    cls = reinterpret_cast<uint8_t*>(tmem_slot + 2);
  }
};

// barriers and tensor memory (all 512 columns)
__device__ __forceinline__ void at_begin(const Bars& bar, int warp, int warps) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < MAX_SLOTS; ++i) { mbar_init(&bar.full[i], 1); mbar_init(&bar.empty[i], 1); }
    mbar_init(bar.res_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&bar.s_full[i], 1); mbar_init(&bar.s_free[i], warps); mbar_init(&bar.p_full[i], warps); mbar_init(&bar.ds_out[i], warps); }
    mbar_init(bar.acc_full, 1);
    *bar.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();      // before tensor memory is taken: see launch_pdl
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(bar.tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}
__device__ __forceinline__ uint32_t at_ready(const Bars& bar) {
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *bar.tmem_slot;
}
// the same and the class list of query tile qt
__device__ __forceinline__ uint32_t at_setup(const AttnParams& p, const Bars& bar, int warp, int lane, int b, int h, int qt) {
  at_begin(bar, warp, EW);
  if (warp == 2 && lane < p.tiles) bar.cls[lane] = (uint8_t)class_of(p, b, h, qt, lane);
  return at_ready(bar);
}
__device__ __forceinline__ void at_teardown(int warp, uint32_t tmem_base) {
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}
__device__ __forceinline__ void give_up(const AttnParams& p, const Bars& bar, int code) {
  if (!*bar.abort_flag) { *bar.abort_flag = 1; atomicExch(p.status, code); }
}

// position in the ring of tiles
struct RingPos {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step(int n) { if (++slot == n) { slot = 0; phase ^= 1u; } }
};
// producer side: wait for the slot, issue the tile
__device__ __forceinline__ bool ring_load(const AttnParams& p, const Bars& bar, RingPos& pos, uint32_t ring, const CUtensorMap* map, int col, int row, int z, int lane, int slots = RING) {
  if (!mbar_wait_warp(&bar.empty[pos.slot], pos.phase ^ 1u, bar.abort_flag)) {
    if (lane == 0) give_up(p, bar, ST_TIMEOUT_PRODUCER);
    return false;
  }
  if (elect_one()) load_tile(ring + (uint32_t)pos.slot * TILE_BYTES, map, &bar.full[pos.slot], col, row, z);
  __syncwarp();
  pos.step(slots);
  return true;
}
__device__ __forceinline__ bool mma_wait(const AttnParams& p, const Bars& bar, uint64_t* b, uint32_t parity, int lane) {
  if (mbar_wait_warp(b, parity, bar.abort_flag)) { tc_fence_after(); return true; }
  if (lane == 0) give_up(p, bar, ST_TIMEOUT_MMA);
  return false;
}
// element-wise side; warp-uniform result
__device__ __forceinline__ bool epi_wait(const AttnParams& p, const Bars& bar, uint64_t* b, uint32_t parity) {
  bool ok = mbar_wait(b, parity, bar.abort_flag);
  if (!ok) give_up(p, bar, ST_TIMEOUT_EPILOGUE);
  ok = __all_sync(0xffffffffu, ok);
  tc_fence_after();
  return ok;
}

// ------------------------------------------------------------------ forward
struct FwdMaps { CUtensorMap q, k, v; };

// 32 scores of the thread's row as packed bf16: bf16(bf16(s * scale) + mask), -inf behind the last column
__device__ __forceinline__ void scaled_scores(const AttnParams& p, uint32_t t_addr, uint32_t cls, const __nv_bfloat16* mrow, int col, uint32_t (&u)[16]) {
  uint32_t v[32];
  tc_ld32(t_addr, v);
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const uint32_t s = pack_bf16x2_rn(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
    u[e] = pack2(mul2f(unpack2(s), both(p.scale)));
  }
  if (cls != 0u && mrow != nullptr) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (col + 8 * c < p.M) {
        const uint4 m = __ldg(reinterpret_cast<const uint4*>(mrow + col + 8 * c));
        u[4 * c] = add2(u[4 * c], m.x); u[4 * c + 1] = add2(u[4 * c + 1], m.y);
        u[4 * c + 2] = add2(u[4 * c + 2], m.z); u[4 * c + 3] = add2(u[4 * c + 3], m.w);
      }
    }
  }
  if (col + 32 > p.M) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (col + 8 * c >= p.M) { u[4 * c] = kNegInf2; u[4 * c + 1] = kNegInf2; u[4 * c + 2] = kNegInf2; u[4 * c + 3] = kNegInf2; }
  }
}

template <int QBIT>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ FwdMaps maps, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  const Bars bar(smem + AT_BARS);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // the query tiles with the most key tiles (a causal map's last ones) start first
  const int bh = (int)blockIdx.x % (p.B * p.heads), qt = p.tiles - 1 - (int)blockIdx.x / (p.B * p.heads);
  const int b = bh / p.heads, h = bh % p.heads, kvh = h / (p.heads / p.kv_heads);
  const uint32_t tmem = at_setup(p, bar, warp, lane, b, h, qt);
  const uint32_t res = smem_u32(smem), ring = res + TILE_BYTES;
  // tensor memory: scores / P in two buffers of 128 columns, O in columns 256..383
  const uint32_t t_o = tmem + 256;
  const int nt = p.tiles;

  if (warp == 0) {
    bool ok = true;
    RingPos pos;
    if (elect_one()) load_tile(res, &maps.q, bar.res_full, h * TILE, qt * TILE, b);
    __syncwarp();
    for (int kt = 0; kt < nt && ok; ++kt)
      if (bar.cls[kt] != 2) ok = ring_load(p, bar, pos, ring, &maps.k, kvh * TILE, kt * TILE, b, lane);
    // K of the next tile comes before V of this one: its product is issued first
    int prev = -1;
    for (int kt = 0; kt < nt && ok; ++kt) {
      if (bar.cls[kt] == 2) continue;
      ok = ring_load(p, bar, pos, ring, &maps.k, kvh * TILE, kt * TILE, b, lane);
      if (ok && prev >= 0) ok = ring_load(p, bar, pos, ring, &maps.v, kvh * TILE, prev * TILE, b, lane);
      prev = kt;
    }
    if (ok && prev >= 0) ring_load(p, bar, pos, ring, &maps.v, kvh * TILE, prev * TILE, b, lane);
  } else if (warp == 1) {
    RingPos pos;
    int n1 = 0;
    for (int kt = 0; kt < nt; ++kt) n1 += bar.cls[kt] != 2;
    bool ok = mma_wait(p, bar, bar.res_full, 0, lane);
    // scores of step t (both passes counted) into buffer t & 1
    auto scores = [&](int t) {
      const int buf = t & 1;
      if (t >= 2 && t - 2 < n1 && !mma_wait(p, bar, &bar.s_free[buf], (uint32_t)((t >> 1) - 1) & 1u, lane)) return false;
      if (!mma_wait(p, bar, &bar.full[pos.slot], pos.phase, lane)) return false;
      const uint32_t kt_addr = ring + (uint32_t)pos.slot * TILE_BYTES;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) tc_mma<false>(tmem + (uint32_t)(buf * TILE), desc_k(res, kk), desc_k(kt_addr, kk), kIdesc, kk > 0 ? 1u : 0u);
        tc_commit<false>(&bar.empty[pos.slot]);
        tc_commit<false>(&bar.s_full[buf]);
      }
      __syncwarp();
      pos.step(RING);
      return true;
    };
    for (int t = 0; t < n1 && ok; ++t) ok = scores(t);
    if (ok && n1 > 0) ok = scores(n1);
    for (int j = 0; j < n1 && ok; ++j) {
      const int t = n1 + j, buf = t & 1;
      if (j + 1 < n1) ok = scores(t + 1);
      ok = ok && mma_wait(p, bar, &bar.p_full[buf], (uint32_t)((t >> 1) - ((n1 + (buf ^ (n1 & 1))) >> 1)) & 1u, lane);
      ok = ok && mma_wait(p, bar, &bar.full[pos.slot], pos.phase, lane);
      if (!ok) break;
      const uint32_t v_addr = ring + (uint32_t)pos.slot * TILE_BYTES, t_p = tmem + (uint32_t)(buf * TILE);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          tc_mma_ta(t_o, t_p + (uint32_t)((kk >> 1) * 32 + (kk & 1) * 8), desc_mn(v_addr, kk), kIdesc | kBMn, (j > 0 || kk > 0) ? 1u : 0u);
        tc_commit<false>(&bar.empty[pos.slot]);
        if (j + 1 == n1) tc_commit<false>(bar.acc_full);
      }
      __syncwarp();
      pos.step(RING);
    }
  } else {
    const int quad = warp & 3, part = (warp - 2) >> 2;
    const int r = quad * 32 + lane, row = qt * TILE + r;
    const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(32 * part);
    const __nv_bfloat16* mrow = p.mask != nullptr && row < p.M ? p.mask + b * p.mb + h * p.mh + (int64_t)row * p.mr : nullptr;
    uint32_t* R = reinterpret_cast<uint32_t*>(smem + AT_EPI) + (warp - 2) * 512;
    float* s_val = reinterpret_cast<float*>(smem + AT_ROWS);             // [4 parts][128] maxima, then [4][128] sums
    bool fine = true;
    // ---- first pass: maximum and sum of the thread's quarter rows
    float m = -INFINITY, sum = 0.f;
    int t = 0;
    for (int kt = 0; kt < nt; ++kt) {
      const uint32_t cls = bar.cls[kt];
      if (cls == 2u) continue;
      const int buf = t & 1;
      fine = fine && epi_wait(p, bar, &bar.s_full[buf], (uint32_t)(t >> 1) & 1u);
      if (fine) {
        uint32_t u[16];
        scaled_scores(p, t_lane + (uint32_t)(buf * TILE), cls, mrow, kt * TILE + 32 * part, u);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.s_free[buf]);
        uint32_t x = max2(u[0], u[1]);
#pragma unroll
        for (int e = 2; e < 16; ++e) x = max2(x, u[e]);
        const float tm = fmaxf(bf16lo_to_f32(x), bf16hi_to_f32(x));
        if (tm > m) {
          sum *= ex2((m - tm) * kLog2e);
          m = tm;
        }
        if (tm != -INFINITY) {      // (a NaN has to reach the sum: the whole row becomes NaN)
          const float k = exp_scale(m);
          const float2 ml = both(-m * k);
          float2 s2[2] = {both(0.f), both(0.f)};
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 z = fma2f(unpack2(u[e]), both(k), ml);
            s2[e & 1] = add2f(s2[e & 1], make_float2(ex2(z.x), ex2(z.y)));
          }
          sum += (s2[0].x + s2[0].y) + (s2[1].x + s2[1].y);
        }
      }
      ++t;
    }
    s_val[part * TILE + r] = m;
    s_val[(4 + part) * TILE + r] = sum;
    at_sync();
    {
      float mp[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) mp[i] = s_val[i * TILE + r];
      m = fmaxf(fmaxf(mp[0], mp[1]), fmaxf(mp[2], mp[3]));
      sum = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) sum += s_val[(4 + i) * TILE + r] * (mp[i] > -INFINITY ? ex2((mp[i] - m) * kLog2e) : 0.f);
    }
    const float inv = 1.0f / sum, k = exp_scale(m);
    const float2 ml = both(-m * k);
    // ---- second pass: probabilities to tensor memory and to the map
    __nv_bfloat16* map = p.map + (int64_t)bh * p.M * p.M;
    // tiles of the map that are written: all, or up to the last one that is not ruled out.  Half of a causal map are zeros that
    // cost as much to write as probabilities: 122 -> 106 us for [1,32,2048,2048], 143 -> 134 for [4,32,1024,1024]
    int written = nt;
    if (p.row_cols != nullptr) {
      while (written > 0 && bar.cls[written - 1] == 2) --written;
      if (part == 0 && row < p.M) p.row_cols[(int64_t)bh * p.M + row] = (uint16_t)min(written * TILE, p.M);
    }
    for (int kt = 0; kt < nt; ++kt) {
      const uint32_t cls = bar.cls[kt];
      const int col = kt * TILE + 32 * part;
      if (cls == 2u) {
        if (p.map != nullptr && kt < written) {      // ruled out: zeros
          const uint4 z = make_uint4(0u, 0u, 0u, 0u);
          for (int i = lane; i < 32 * 4; i += 32) {
            const int zr = qt * TILE + quad * 32 + (i >> 2), zc = col + 8 * (i & 3);
            if (zr < p.M && zc < p.M) *reinterpret_cast<uint4*>(map + (int64_t)zr * p.M + zc) = z;
          }
        }
        continue;
      }
      const int buf = t & 1;
      fine = fine && epi_wait(p, bar, &bar.s_full[buf], (uint32_t)(t >> 1) & 1u);
      if (fine) {
        uint32_t u[16];
        scaled_scores(p, t_lane + (uint32_t)(buf * TILE), cls, mrow, col, u);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float2 z = fma2f(unpack2(u[e]), both(k), ml);
          u[e] = pack2(mul2f(make_float2(ex2(z.x), ex2(z.y)), both(inv)));
        }
        // over the scores of this quarter (all read by now): 32 columns as 16 words
        tc_st16(t_lane + (uint32_t)(buf * TILE), u);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.p_full[buf]);
        if (p.map != nullptr) {
#pragma unroll
          for (int e = 0; e < 4; ++e) *reinterpret_cast<uint4*>(R + gd_chunk(lane, e)) = make_uint4(u[4 * e], u[4 * e + 1], u[4 * e + 2], u[4 * e + 3]);
          __syncwarp();
          flush_clipped(R, map, qt * TILE + quad * 32, p.M, p.M, col, p.M, lane);
          __syncwarp();
        }
      }
      ++t;
    }
    // ---- O: bf16 and its per-channel codes
    fine = fine && t > 0 && epi_wait(p, bar, bar.acc_full, 0);
    if (fine) {
      const int64_t ld = (int64_t)p.heads * TILE;
      uint32_t acc[32], w[BlockGeo<QBIT>::NW], o[16];
      const int n = h * TILE + 32 * part;
      tc_ld32(t_lane + 256u, acc);
      put_row_bf16(R, lane, acc);
      __syncwarp();
      flush_clipped(R, p.out0 + (int64_t)b * p.M * ld, qt * TILE + quad * 32, p.M, ld, n, (int)ld, lane);
      if (p.codes != nullptr && row < p.M) {
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e] = pack_bf16x2_rn(__uint_as_float(acc[2 * e]), __uint_as_float(acc[2 * e + 1]));
#pragma unroll
        for (int i = 0; i < BlockGeo<QBIT>::NW; ++i) w[i] = 0u;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const uint32_t s2 = __ldg(reinterpret_cast<const uint32_t*>(p.code_scale + n + 2 * e));
          put_code<QBIT>(w, 2 * e, fastq_code_bits<QBIT>(bf16lo_to_f32(o[e]), fastq_scale<QBIT>(__frcp_rn(bf16lo_to_f32(s2)))) & BlockGeo<QBIT>::CM);
          put_code<QBIT>(w, 2 * e + 1, fastq_code_bits<QBIT>(bf16hi_to_f32(o[e]), fastq_scale<QBIT>(__frcp_rn(bf16hi_to_f32(s2)))) & BlockGeo<QBIT>::CM);
        }
        store_block_words<QBIT>(p.codes + (((int64_t)b * p.M + row) * ld + n) * QBIT / 8, w);
      }
    }
  }
  at_teardown(warp, tmem);
}

// ------------------------------------------------------------------ backward, q side
// maps: dO (hidden layout), V, K (hidden layout), P (the restored map [B * heads, M, M])
struct BwdQMaps { CUtensorMap g, v, k, p; };

// dS leaves through the ring slot of the P that it was made from: what a staging tile of its own would take buys two more slots, so that
// two steps of three tiles are in flight ([1,32,2048,2048] causal, cold: 111.8 -> 105.5 us).
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_bwd_q_kernel(const __grid_constant__ BwdQMaps maps, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  const Bars bar(smem + Q_BARS);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int bh = (int)blockIdx.x % (p.B * p.heads), qt = p.tiles - 1 - (int)blockIdx.x / (p.B * p.heads);
  const int b = bh / p.heads, h = bh % p.heads, kvh = h / (p.heads / p.kv_heads);
  const uint32_t tmem = at_setup(p, bar, warp, lane, b, h, qt);
  const uint32_t res = smem_u32(smem), ring = res + TILE_BYTES;
  // tensor memory: dP / dS in two buffers of 128 columns, dQ in columns 256..383
  const uint32_t t_acc = tmem + 256;
  const int nt = p.tiles;

  if (warp == 0) {
    bool ok = true;
    RingPos pos;
    if (elect_one()) load_tile(res, &maps.g, bar.res_full, h * TILE, qt * TILE, b);
    __syncwarp();
    for (int kt = 0; kt < nt && ok; ++kt) {
      if (bar.cls[kt] == 2) continue;
      ok = ring_load(p, bar, pos, ring, &maps.v, kvh * TILE, kt * TILE, b, lane, Q_RING);
      ok = ok && ring_load(p, bar, pos, ring, &maps.p, kt * TILE, qt * TILE, bh, lane, Q_RING);
    }
    // a step takes three of the six slots, so the P of step j lies where that of step j - 2 was: its dS has to be out
    int j = 0;
    for (int kt = 0; kt < nt && ok; ++kt) {
      if (bar.cls[kt] == 2) continue;
      ok = ring_load(p, bar, pos, ring, &maps.v, kvh * TILE, kt * TILE, b, lane, Q_RING);
      if (ok && j >= 2 && !mbar_wait_warp(&bar.ds_out[j & 1], (uint32_t)((j >> 1) - 1) & 1u, bar.abort_flag)) {
        if (lane == 0) give_up(p, bar, ST_TIMEOUT_PRODUCER);
        ok = false;
      }
      ok = ok && ring_load(p, bar, pos, ring, &maps.p, kt * TILE, qt * TILE, bh, lane, Q_RING);
      ok = ok && ring_load(p, bar, pos, ring, &maps.k, kvh * TILE, kt * TILE, b, lane, Q_RING);
      ++j;
    }
  } else if (warp == 1) {
    RingPos pos;
    int n1 = 0;
    for (int kt = 0; kt < nt; ++kt) n1 += bar.cls[kt] != 2;
    bool ok = mma_wait(p, bar, bar.res_full, 0, lane);
    // dP = dO V^T of step t (both passes counted) into buffer t & 1
    auto grad_map = [&](const RingPos& at, int t) {
      if (!mma_wait(p, bar, &bar.full[at.slot], at.phase, lane)) return false;
      const uint32_t v_addr = ring + (uint32_t)at.slot * TILE_BYTES;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) tc_mma<false>(tmem + (uint32_t)((t & 1) * TILE), desc_k(res, kk), desc_k(v_addr, kk), kIdesc, kk > 0 ? 1u : 0u);
        tc_commit<false>(&bar.empty[at.slot]);
        tc_commit<false>(&bar.s_full[t & 1]);
      }
      __syncwarp();
      return true;
    };
    // first pass, slots of step t: V, P.  A step that has been read frees its buffer and its P
    auto step_read = [&](int t) {
      if (!mma_wait(p, bar, &bar.s_free[t & 1], (uint32_t)(t >> 1) & 1u, lane)) return false;
      if (elect_one()) mbar_arrive(&bar.empty[(2 * t + 1) % Q_RING]);
      __syncwarp();
      return true;
    };
    for (int t = 0; t < n1 && ok; ++t) {
      ok = (t < 2 || step_read(t - 2)) && grad_map(pos, t);
      pos.step(Q_RING); pos.step(Q_RING);
    }
    for (int t = n1 > 1 ? n1 - 2 : 0; t < n1 && ok; ++t) ok = step_read(t);
    // second pass, slots of step j: V, P, K
    RingPos pv = pos;
    if (ok && n1 > 0) ok = grad_map(pv, n1);
    for (int j = 0; j < n1 && ok; ++j) {
      const int t = n1 + j, buf = t & 1;
      pv.step(Q_RING); pv.step(Q_RING); pv.step(Q_RING);
      if (j + 1 < n1) ok = grad_map(pv, t + 1);
      ok = ok && mma_wait(p, bar, &bar.p_full[buf], (uint32_t)((t >> 1) - ((n1 + (buf ^ (n1 & 1))) >> 1)) & 1u, lane);
      pos.step(Q_RING);                          // V
      const int p_slot = pos.slot;
      pos.step(Q_RING);
      ok = ok && mma_wait(p, bar, &bar.full[pos.slot], pos.phase, lane);
      if (!ok) break;
      const uint32_t k_addr = ring + (uint32_t)pos.slot * TILE_BYTES, t_s = tmem + (uint32_t)(buf * TILE);
      if (elect_one()) {
        mbar_arrive(&bar.empty[p_slot]);         // (dS still leaves through it: the producer waits for that too)
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          tc_mma_ta(t_acc, t_s + (uint32_t)((kk >> 1) * 32 + (kk & 1) * 8), desc_mn(k_addr, kk), kIdesc | kBMn, (j > 0 || kk > 0) ? 1u : 0u);
        tc_commit<false>(&bar.empty[pos.slot]);
        if (j + 1 == n1) tc_commit<false>(bar.acc_full);
      }
      __syncwarp();
      pos.step(Q_RING);
    }
  } else {
    const int quad = warp & 3, part = (warp - 2) >> 2;
    const int r = quad * 32 + lane;
    const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(32 * part);
    float* s_val = reinterpret_cast<float*>(smem + Q_ROWS);
    bool fine = true;
    // 16-byte chunk c of this warp's quarter of row rr (a 128-byte row of a swizzled sub-tile holds two quarters)
    auto chunk_at = [&](uint8_t* tile, int rr, int c) {
      return reinterpret_cast<uint4*>(tile + (part >> 1) * (TILE_BYTES / 2) + rr * 128 + (((4 * (part & 1) + c) ^ (rr & 7)) << 4));
    };
    // ---- D = rowsum of the bf16 products P * bf16(dP)
    float2 d2 = both(0.f);
    RingPos pp;                                  // the P of each step
    pp.slot = 1;
    int t = 0;
    for (int kt = 0; kt < nt; ++kt) {
      if (bar.cls[kt] == 2) continue;
      const int buf = t & 1;
      fine = fine && epi_wait(p, bar, &bar.full[pp.slot], pp.phase);
      fine = fine && epi_wait(p, bar, &bar.s_full[buf], (uint32_t)(t >> 1) & 1u);
      if (fine) {
        uint8_t* pt = smem + TILE_BYTES * (1 + pp.slot);
        uint32_t acc[32];
        tc_ld32(t_lane + (uint32_t)(buf * TILE), acc);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint4 q4 = *chunk_at(pt, r, e);
          const uint32_t pw[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
            d2 = add2f(d2, unpack2(mul2(pw[i], pack_bf16x2_rn(__uint_as_float(acc[8 * e + 2 * i]), __uint_as_float(acc[8 * e + 2 * i + 1])))));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.s_free[buf]);
      }
      pp.step(Q_RING); pp.step(Q_RING);
      ++t;
    }
    // (as (0 + 1) + (2 + 3) of the four parts)
    if (part & 1) s_val[(part >> 1) * TILE + r] = d2.x + d2.y;
    at_sync();
    if (!(part & 1)) s_val[(part >> 1) * TILE + r] += d2.x + d2.y;
    at_sync();
    const float2 minus_d = both(-(s_val[r] + s_val[TILE + r]));
    // ---- dS = bf16(bf16((bf16(dP) - D) * P) * scale)
    __nv_bfloat16* ds = p.map + (int64_t)bh * p.M * p.M;
    // pp stands one slot behind the first V of this pass: its P
    int j = 0;
    for (int kt = 0; kt < nt; ++kt) {
      if (bar.cls[kt] == 2) continue;
      const int buf = t & 1;
      fine = fine && epi_wait(p, bar, &bar.full[pp.slot], pp.phase);
      fine = fine && epi_wait(p, bar, &bar.s_full[buf], (uint32_t)(t >> 1) & 1u);
      if (fine) {
        uint8_t* pt = smem + TILE_BYTES * (1 + pp.slot);
        uint32_t w[16], acc[32];
        tc_ld32(t_lane + (uint32_t)(buf * TILE), acc);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint4 q4 = *chunk_at(pt, r, e);
          const uint32_t pw[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t g = pack_bf16x2_rn(__uint_as_float(acc[8 * e + 2 * i]), __uint_as_float(acc[8 * e + 2 * i + 1]));
            const uint32_t s = pack2(mul2f(add2f(unpack2(g), minus_d), unpack2(pw[i])));
            w[4 * e + i] = pack2(mul2f(unpack2(s), both(p.scale)));
          }
        }
        tc_st16(t_lane + (uint32_t)(buf * TILE), w);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.p_full[buf]);
#pragma unroll
        for (int e = 0; e < 4; ++e) *chunk_at(pt, r, e) = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
        __syncwarp();
        // eight lanes read two rows whose chunks the swizzle puts on different banks
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int rr = quad * 32 + 8 * k + (lane >> 3) + 4 * ((lane >> 2) & 1), row = qt * TILE + rr, c = kt * TILE + 32 * part + 8 * (lane & 3);
          const uint4 v = *chunk_at(pt, rr, lane & 3);
          if (row < p.M && c < p.M) *reinterpret_cast<uint4*>(ds + (int64_t)row * p.M + c) = v;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the next tile of this slot comes by TMA
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.ds_out[j & 1]);
      }
      pp.step(Q_RING); pp.step(Q_RING); pp.step(Q_RING);
      ++t;
      ++j;
    }
    fine = fine && j > 0 && epi_wait(p, bar, bar.acc_full, 0);
    if (fine) {
      // through the dO tile: its last readers were the products that came before the last of dQ
      uint32_t* R = reinterpret_cast<uint32_t*>(smem) + (warp - 2) * 512;
      const int64_t ld = (int64_t)p.heads * TILE;
      uint32_t acc[32];
      tc_ld32(t_lane + 256u, acc);
      put_row_bf16(R, lane, acc);
      __syncwarp();
      flush_clipped(R, p.out0 + (int64_t)b * p.M * ld, qt * TILE + quad * 32, p.M, ld, h * TILE + 32 * part, (int)ld, lane);
    }
  }
  at_teardown(warp, tmem);
}

// ------------------------------------------------------------------ backward, kv side
// maps: P, dS ([B * heads, M, M]), dO, Q (hidden layout)
struct BwdKvMaps { CUtensorMap p, s, g, q; };

// the query tiles that do not rule key tile kt out, one bit each (all lanes get all of them)
__device__ __forceinline__ uint32_t live_query_tiles(const AttnParams& p, int b, int h, int kt, int lane) {
  return __ballot_sync(0xffffffffu, lane < p.tiles && class_of(p, b, h, lane, kt) != 2u);
}
// item -> batch, key/value head, key tile.  The first key tiles have the most query tiles under a causal mask: they come first
struct KvItem {
  int b, kvh, kt;
  __device__ __forceinline__ KvItem(const AttnParams& p, int item) {
    const int bk = item % (p.B * p.kv_heads);
    kt = item / (p.B * p.kv_heads); b = bk / p.kv_heads; kvh = bk % p.kv_heads;
  }
};
// The items of a block: one of every `gridDim.x`, taken in turn from either end, so that long and short ones add up to the same.
// All roles walk the same list.
__device__ __forceinline__ int kv_item(int round) {
  const int g = (int)gridDim.x;
  return round * g + ((round & 1) ? g - 1 - (int)blockIdx.x : (int)blockIdx.x);
}

// MANY: a block per SM and more items than blocks: the loads of the next item run while the gradients of this one leave, which is
// why each item has accumulators of its own (dV and dK, two sets).  Without it a block has one item; a list of one would cost 0.1 to 0.5 us
// of its fixed share.  Single launches, cold, us, a block per item / MANY: [1,32,2048,2048] causal, 512 items 73.5 / 65.2; 160 items
// [5,32,128,128] 14.7 / 12.9; 192 [3,32,256,256] 16.1 / 14.2; 256 [1,32,1024,1024] 25.2 / 23.0; 288 [1,32,1152,1152] 28.9 / 26.3.  Items of
// four heads each (8 key/value heads) keep their loads under way by themselves: 160 [5,32,512,512] 52.6 / 50.7 without a mask, 192 causal 35.5 / 35.1,
// 256 [4,32,1024,1024] 68.4 / 68.5, 256 [8,32,512,512] causal 46.2 / 48.1, 288 without a mask 75.5 / 75.6.
// Both backward kernels between a pair of events, four slots and a block per item / six slots and this: [1,32,2048,2048] causal 193 / 179, [4,32,1024,1024]
// 250 / 232 (with 8 key/value heads 198 / 196), [2,32,696,696] 83.0 / 75.9, [1,32,2048,2048] without a mask 349 / 318, [3,32,256,256] 35.8 / 35.1;
// short rows with 8 key/value heads lose by the q kernel's slots: [4,32,512,512] 101.6 / 103.2 without a mask (the q kernel 60.0 / 61.4), 79.8 / 80.3 causal.
template <bool MANY>
__global__ void __launch_bounds__(KV_THREADS, 1)
attn_bwd_kv_kernel(const __grid_constant__ BwdKvMaps maps, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  const Bars bar(smem + KV_BARS);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rep = p.heads / p.kv_heads, items = p.tiles * p.B * p.kv_heads;
  // -1: there are no more of them
  auto item_of = [&](int round) {
    if (!MANY) return round == 0 ? (int)blockIdx.x : -1;
    const int item = kv_item(round);
    return item < items ? item : -1;
  };
  at_begin(bar, warp, KV_WARPS);
  const uint32_t tmem = at_ready(bar);
  const uint32_t ring = smem_u32(smem);
  constexpr int SLOTS = KV_SLOTS;

  if (warp == 0) {
    bool ok = true;
    RingPos pos;
    int item = item_of(0);
    const KvItem first(p, item);
    uint32_t next = live_query_tiles(p, first.b, first.kvh * rep, first.kt, lane);
    for (int round = 0; item >= 0 && ok; ++round) {
      const KvItem w(p, item);
      const uint32_t live = next;
      item = item_of(round + 1);
      bool asked = false;
      // the classes of the next item are looked up while the first tiles of this one are on their way
      auto ask = [&]() {
        if (!asked && item >= 0) { const KvItem n(p, item); next = live_query_tiles(p, n.b, n.kvh * rep, n.kt, lane); }
        asked = true;
      };
      for (int g = 0; g < rep && ok; ++g) {
        const int h = w.kvh * rep + g, bh = w.b * p.heads + h;
        for (uint32_t left = live; left != 0u && ok; left &= left - 1u) {
          const int qt = __ffs(left) - 1;
          ok = ring_load(p, bar, pos, ring, &maps.p, w.kt * TILE, qt * TILE, bh, lane, SLOTS) &&
               ring_load(p, bar, pos, ring, &maps.g, h * TILE, qt * TILE, w.b, lane, SLOTS) &&
               ring_load(p, bar, pos, ring, &maps.s, w.kt * TILE, qt * TILE, bh, lane, SLOTS) &&
               ring_load(p, bar, pos, ring, &maps.q, h * TILE, qt * TILE, w.b, lane, SLOTS);
          ask();
        }
      }
      ask();
    }
  } else if (warp == 1) {
    RingPos pos;
    bool ok = true;
    int used = 0;                                   // items with products so far
    for (int round = 0, item; (item = item_of(round)) >= 0 && ok; ++round) {
      const KvItem w(p, item);
      const int steps = 2 * rep * __popc(live_query_tiles(p, w.b, w.kvh * rep, w.kt, lane));      // dV from P and dO, dK from dS and Q
      if (steps == 0) continue;
      const int set = used & 1;
      if (used >= 2) ok = mma_wait(p, bar, &bar.s_free[set], (uint32_t)((used >> 1) - 1) & 1u, lane);
      for (int i = 0; i < steps && ok; ++i) {
        RingPos pb = pos;
        pb.step(SLOTS);
        ok = mma_wait(p, bar, &bar.full[pos.slot], pos.phase, lane) && mma_wait(p, bar, &bar.full[pb.slot], pb.phase, lane);
        if (!ok) break;
        const uint32_t a_addr = ring + (uint32_t)pos.slot * TILE_BYTES, b_addr = ring + (uint32_t)pb.slot * TILE_BYTES;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma<false>(tmem + (uint32_t)((2 * set + (i & 1)) * TILE), desc_mn(a_addr, kk), desc_mn(b_addr, kk), kIdesc | kAMn | kBMn, (i > 1 || kk > 0) ? 1u : 0u);
          tc_commit<false>(&bar.empty[pos.slot]);
          tc_commit<false>(&bar.empty[pb.slot]);
          if (i + 1 == steps) tc_commit<false>(&bar.s_full[set]);
        }
        __syncwarp();
        pos = pb;
        pos.step(SLOTS);
      }
      ++used;
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t t_lane = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(64 * half);
    uint32_t* R = reinterpret_cast<uint32_t*>(smem + KV_EPI) + (warp - 2) * 512;
    const int64_t ld = (int64_t)p.kv_heads * TILE;
    bool fine = true;
    int used = 0;
    for (int round = 0, item; (item = item_of(round)) >= 0 && fine; ++round) {
      const KvItem w(p, item);
      // keys that no query row attends to get zero gradients
      const bool any = live_query_tiles(p, w.b, w.kvh * rep, w.kt, lane) != 0u;
      const int set = used & 1;
      fine = !any || epi_wait(p, bar, &bar.s_full[set], (uint32_t)(used >> 1) & 1u);
      if (!fine) break;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t acc[32];
        if (any) {
          tc_ld32(t_lane + (uint32_t)((2 * set + (c >> 1)) * TILE + 32 * (c & 1)), acc);
          if (c == 3) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar.s_free[set]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) acc[e] = 0u;
        }
        put_row_bf16(R, lane, acc);
        __syncwarp();
        flush_clipped(R, (c < 2 ? p.out1 : p.out0) + (int64_t)w.b * p.M * ld, w.kt * TILE + quad * 32, p.M, ld, w.kvh * TILE + 64 * half + 32 * (c & 1), (int)ld, lane);
        __syncwarp();
      }
      if (any) ++used;
    }
  }
  at_teardown(warp, tmem);
}

// ------------------------------------------------------------------ host side
static bool map_3d(CUtensorMap* m, const void* ptr, int64_t cols, int64_t rows, int64_t depth) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)depth};
  cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)(cols * rows) * 2};
  cuuint32_t box[3] = {64u, (cuuint32_t)TILE, 1u};
  cuuint32_t estr[3] = {1u, 1u, 1u};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename K>
static int at_prepare(K kern, int smem, bool (&done)[64]) {
  const int slot = current_device_slot();
  if (slot >= 0 && done[slot]) return HYC_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    hyc_set_last_cuda_error((int)cudaGetLastError());
    return HYC_ERR_LAUNCH;
  }
  if (slot >= 0) done[slot] = true;
  return HYC_OK;
}

static int at_check(int B, int M, int heads, int kv_heads, int head_dim) {
  if (head_dim != TILE) return HYC_ERR_UNSUPPORTED;
  if (B < 1 || M < 1 || M % 8 != 0 || heads < 1 || kv_heads < 1 || heads % kv_heads != 0) return HYC_ERR_SHAPE;
  if (M > MAX_TILES * TILE) return HYC_ERR_UNSUPPORTED;
  return HYC_OK;
}

template <int QBIT>
static int launch_fwd(const FwdMaps& maps, const AttnParams& p, cudaStream_t st) {
  static bool done[64] = {false};
  if (const int rc = at_prepare(attn_fwd_kernel<QBIT>, AT_SMEM, done)) return rc;
  launch_pdl(attn_fwd_kernel<QBIT>, dim3((unsigned)(p.tiles * p.B * p.heads)), dim3(AT_THREADS), AT_SMEM, st, maps, p);
  HYC_CHECK_LAUNCH();
  return HYC_OK;
}

}  // namespace at
}  // namespace hyc

using namespace hyc;
using namespace hyc::at;

extern "C" HYC_API size_t hyc_attn_mask_class_bytes(int mask_batch, int mask_heads, int M) {
  const size_t t = (size_t)(M + TILE - 1) / TILE;
  return (size_t)mask_batch * mask_heads * t * t * sizeof(TileClass);
}

extern "C" HYC_API int hyc_attn_mask_class(const void* mask, int64_t stride_b, int64_t stride_h, int64_t stride_row, int mask_batch, int mask_heads,
                                           int M, void* out, void* stream) {
  if (!mask || !out) return HYC_ERR_NULL;
  if (mask_batch < 1 || mask_heads < 1 || M < 1 || M % 8 != 0 || M > MAX_TILES * TILE) return HYC_ERR_SHAPE;
  if (!aligned(mask, 16) || !aligned(out, 16) || ((stride_b | stride_h | stride_row) & 7)) return HYC_ERR_ALIGN;
  const int t = (M + TILE - 1) / TILE;
  launch_pdl(mask_class_kernel, dim3(t, t, mask_batch * mask_heads), dim3(256), 0, (cudaStream_t)stream, 
      (const __nv_bfloat16*)mask, stride_b, stride_h, stride_row, M, t, mask_heads, (TileClass*)out);
  HYC_CHECK_LAUNCH();
  return HYC_OK;
}

extern "C" HYC_API int hyc_attn_fwd_tcgen05(
    const void* q, const void* k, const void* v, int B, int M, int heads, int kv_heads, int head_dim, float scale,
    const void* mask, int64_t mask_b, int64_t mask_h, int64_t mask_row, const void* cls, int64_t cls_b, int64_t cls_h,
    void* map, void* o, const void* o_scale, void* o_codes, int q_bit, int* status, void* stream) {
  return hyc_attn_fwd_cols_tcgen05(q, k, v, B, M, heads, kv_heads, head_dim, scale, mask, mask_b, mask_h, mask_row, cls, cls_b, cls_h, map, nullptr, o,
                                   o_scale, o_codes, q_bit, status, stream);
}

extern "C" HYC_API int hyc_attn_fwd_cols_tcgen05(
    const void* q, const void* k, const void* v, int B, int M, int heads, int kv_heads, int head_dim, float scale,
    const void* mask, int64_t mask_b, int64_t mask_h, int64_t mask_row, const void* cls, int64_t cls_b, int64_t cls_h,
    void* map, uint16_t* row_cols, void* o, const void* o_scale, void* o_codes, int q_bit, int* status, void* stream) {
  if (!q || !k || !v || !o || !status || (o_codes != nullptr) != (o_scale != nullptr) || (cls && !mask)) return HYC_ERR_NULL;
  if (const int rc = at_check(B, M, heads, kv_heads, head_dim)) return rc;
  if (o_codes && q_bit != 2 && q_bit != 4 && q_bit != 8) return HYC_ERR_QBIT;
  const void* al[] = {q, k, v, o, map, mask, cls, o_codes, o_scale};
  for (const void* x : al) if (x && !aligned(x, 16)) return HYC_ERR_ALIGN;
  if (mask && ((mask_b | mask_h | mask_row) & 7)) return HYC_ERR_ALIGN;
  FwdMaps maps;
  if (!map_3d(&maps.q, q, (int64_t)heads * TILE, M, B) || !map_3d(&maps.k, k, (int64_t)kv_heads * TILE, M, B) ||
      !map_3d(&maps.v, v, (int64_t)kv_heads * TILE, M, B)) return HYC_ERR_UNSUPPORTED;
  AttnParams p = {};
  p.B = B; p.M = M; p.heads = heads; p.kv_heads = kv_heads; p.tiles = (M + TILE - 1) / TILE; p.scale = scale;
  p.mask = (const __nv_bfloat16*)mask; p.mb = mask_b; p.mh = mask_h; p.mr = mask_row;
  p.cls = (const TileClass*)cls; p.cls_b = cls_b; p.cls_h = cls_h;
  p.out0 = (__nv_bfloat16*)o; p.map = (__nv_bfloat16*)map;
  p.code_scale = (const __nv_bfloat16*)o_scale; p.codes = (uint8_t*)o_codes;
  p.row_cols = map ? row_cols : nullptr;
  p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  if (q_bit == 2) return launch_fwd<2>(maps, p, st);
  if (q_bit == 8) return launch_fwd<8>(maps, p, st);
  return launch_fwd<4>(maps, p, st);
}

extern "C" HYC_API int hyc_attn_bwd_tcgen05(
    const void* q, const void* k, const void* v, const void* grad_o, const void* map, void* grad_s, int B, int M, int heads, int kv_heads,
    int head_dim, float scale, const void* cls, int64_t cls_b, int64_t cls_h, void* grad_q, void* grad_k, void* grad_v, int* status, void* stream) {
  if (!q || !k || !v || !grad_o || !map || !grad_s || !grad_q || !grad_k || !grad_v || !status) return HYC_ERR_NULL;
  if (const int rc = at_check(B, M, heads, kv_heads, head_dim)) return rc;
  const void* al[] = {q, k, v, grad_o, map, grad_s, grad_q, grad_k, grad_v, cls};
  for (const void* x : al) if (x && !aligned(x, 16)) return HYC_ERR_ALIGN;
  const int64_t hd = (int64_t)heads * TILE, kd = (int64_t)kv_heads * TILE, BH = (int64_t)B * heads;
  BwdQMaps mq;
  BwdKvMaps mk;
  if (!map_3d(&mq.g, grad_o, hd, M, B) || !map_3d(&mq.v, v, kd, M, B) || !map_3d(&mq.k, k, kd, M, B) || !map_3d(&mq.p, map, M, M, BH) ||
      !map_3d(&mk.s, grad_s, M, M, BH) || !map_3d(&mk.q, q, hd, M, B)) return HYC_ERR_UNSUPPORTED;
  mk.p = mq.p; mk.g = mq.g;
  AttnParams p = {};
  p.B = B; p.M = M; p.heads = heads; p.kv_heads = kv_heads; p.tiles = (M + TILE - 1) / TILE; p.scale = scale;
  // one class list per key tile serves all heads of a group: with a mask per head and grouped heads nothing is skipped
  if (cls && !(cls_h != 0 && heads != kv_heads)) { p.cls = (const TileClass*)cls; p.cls_b = cls_b; p.cls_h = cls_h; }
  p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  static bool done_q[64] = {false}, done_kv[2][64] = {};
  if (const int rc = at_prepare(attn_bwd_q_kernel, Q_SMEM, done_q)) return rc;
  if (const int rc = at_prepare(attn_bwd_kv_kernel<false>, KV_SMEM, done_kv[0])) return rc;
  if (const int rc = at_prepare(attn_bwd_kv_kernel<true>, KV_SMEM, done_kv[1])) return rc;
  p.out0 = (__nv_bfloat16*)grad_q; p.map = (__nv_bfloat16*)grad_s;
  launch_pdl(attn_bwd_q_kernel, dim3((unsigned)(p.tiles * B * heads)), dim3(AT_THREADS), Q_SMEM, st, mq, p);
  HYC_CHECK_LAUNCH();
  p.out0 = (__nv_bfloat16*)grad_k; p.out1 = (__nv_bfloat16*)grad_v;
  // up to an item per SM: a block each (measured at the kernel)
  const int items = p.tiles * B * kv_heads, sms = num_sms();
  if (items <= sms) launch_pdl(attn_bwd_kv_kernel<false>, dim3((unsigned)items), dim3(KV_THREADS), KV_SMEM, st, mk, p);
  else launch_pdl(attn_bwd_kv_kernel<true>, dim3((unsigned)sms), dim3(KV_THREADS), KV_SMEM, st, mk, p);
  HYC_CHECK_LAUNCH();
  return HYC_OK;
}
