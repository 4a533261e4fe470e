// Shared parts of the tcgen05 GEMM kernels: launch parameters, PTX wrappers, the element-wise epilogues and the
// tensor-map encoder.
#pragma once
#include "hyc_common.cuh"
#include <cuda.h>

namespace hyc {
namespace tc {

constexpr int BM = 128, BN = 256, BK = 64;       // per CTA: 128 rows x 256 columns of accumulator
constexpr int STAGE_A_BYTES = BM * BK * 2;
// PAIR: two CTAs share a 256 x 256 tile, each loads 128 columns of the B block (6 stages of 32 KB);
// otherwise a CTA has a 128 x 256 tile of its own and loads the whole B block (4 stages of 48 KB)
template <bool PAIR> struct Geo {
  static constexpr int TILE_M = PAIR ? 2 * BM : BM;
  static constexpr int B_COLS = PAIR ? BN / 2 : BN;
  static constexpr int STAGE_B_BYTES = B_COLS * BK * 2;
  static constexpr int STAGE_BYTES = STAGE_A_BYTES + STAGE_B_BYTES;
  static constexpr int STAGES = PAIR ? 6 : 4;
};
constexpr int MAX_STAGES = 8;
constexpr int PIPE_BYTES = 6 * (STAGE_A_BYTES + (BN / 2) * BK * 2);
static_assert(PIPE_BYTES == Geo<true>::STAGES * Geo<true>::STAGE_BYTES && PIPE_BYTES == Geo<false>::STAGES * Geo<false>::STAGE_BYTES,
              "both forms use the same amount of shared memory");
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int TMEM_COLS = 512;
// epilogue scratch: 32 KB of tiles followed by BN floats of per-column constants.
//   per epilogue warp two [32 rows][32 columns] bf16 tiles (LoRA terms and residual in, results out), then
//   STORE BN quantizer constants, GATEUP two vectors of BN/2, GRADDOWN two bf16 scale vectors of BN
constexpr int EPI_SMEM_BYTES = 2 * BN * 16 * 4 + BN * 4;
constexpr int SMEM_BYTES = 1024 + PIPE_BYTES + EPI_SMEM_BYTES + 256;
constexpr uint32_t SPIN_LIMIT = 1u << 22;

enum { EPI_STORE = 0, EPI_GATEUP = 1, EPI_GRADDOWN = 2 };
enum { ST_OK = 0, ST_TIMEOUT_PRODUCER = 1, ST_TIMEOUT_MMA = 2, ST_TIMEOUT_EPILOGUE = 3 };

struct LoraTerm {
  const __nv_bfloat16* xa;    // [M, 16] row-major, or null
  const __nv_bfloat16* bt;    // element (col, r) at bt[col * ld_col + r * ld_r]
  int64_t ld_col, ld_r;
};

// tensor maps of a launch: up to four K segments (A, B) or three weights side by side; n: the B operands again in boxes of
// 64 rows, for the half-width tiles of a K-major B
struct Maps { CUtensorMap a[4], b[4], n[4]; };

struct Params {
  int M, N, K1, K2, K3, K4;   // K2, K3, K4 > 0: further (A, B) pairs accumulated into the same tile
  int epi, q_bit;
  LoraTerm l0, l1, l2;        // STORE: l0/l1 added; GATEUP: l0 gate, l1 up; GRADDOWN: l0 grad LoRA, l1 gate, l2 up
  const __nv_bfloat16* residual;   // STORE, [M, N] or null
  __nv_bfloat16* out0;        // STORE: D ; GATEUP: o ; GRADDOWN: o (hadamard)
  __nv_bfloat16* out1;        // GRADDOWN: grad_gate
  __nv_bfloat16* out2;        // GRADDOWN: grad_up
  __nv_bfloat16* dbg1;        // GATEUP: optional bf16 copy of gate_main
  __nv_bfloat16* dbg2;        // GATEUP: optional bf16 copy of up_main
  uint8_t* q1;                // GATEUP: out ; GRADDOWN: in
  uint8_t* q2;
  const __nv_bfloat16* s1;    // per-channel scales [N]
  const __nv_bfloat16* s2;
  const __nv_bfloat16* lpre1; // GRADDOWN: optional precomputed LoRA terms bf16(xa1 B1^T), bf16(xa2 B2^T), [M, ld_pre]
  const __nv_bfloat16* lpre2;
  int64_t ld_pre;
  // STORE with up to three weights side by side along N (q/k/v): columns [0, g_end0) belong to out0/q1/s1/l0,
  // [g_end0, g_end1) to g1 and the rest to g2; their weights are mapB1, mapB2, mapB3.  One weight: g_end0 = g_end1 = N
  int g_end0, g_end1;
  struct Group { __nv_bfloat16* out; uint8_t* q; const __nv_bfloat16* s; LoraTerm l; } g1, g2;
  // Column tiles: the first n_wide are TILE_N columns wide, the rest half of that
  int n_wide;
  int stages, stage_bytes;    // ring of the main loop
  bool fixed_order;           // for the launch: K is not split
  int* status;
#ifdef HYC_TC_PROF
  long long* prof;            // debug builds only: clock64 stamps of CTA 0, [role][tile][8]
#endif
};

// where the columns of one STORE tile go
struct StoreView {
  __nv_bfloat16* out;
  __nv_bfloat16* main;              // optional bf16 copy of the main branch
  uint8_t* q;
  const __nv_bfloat16* s;
  const __nv_bfloat16* residual;
  LoraTerm l0, l1;
  int64_t ld;                       // columns of the group
  int group, n0;                    // group number, first column inside the group
};
__device__ __forceinline__ StoreView store_view(const Params& p, int n0) {
  StoreView v;
  v.main = p.dbg1; v.residual = p.residual; v.l1 = p.l1;
  if (n0 < p.g_end0) {
    v.out = p.out0; v.q = p.q1; v.s = p.s1; v.l0 = p.l0; v.ld = p.g_end0; v.n0 = n0; v.group = 0;
  } else if (n0 < p.g_end1) {
    v.out = p.g1.out; v.q = p.g1.q; v.s = p.g1.s; v.l0 = p.g1.l; v.ld = p.g_end1 - p.g_end0; v.n0 = n0 - p.g_end0; v.group = 1;
  } else {
    v.out = p.g2.out; v.q = p.g2.q; v.s = p.g2.s; v.l0 = p.g2.l; v.ld = p.N - p.g_end1; v.n0 = n0 - p.g_end1; v.group = 2;
  }
  return v;
}

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Dynamic shared memory from the next 1024-byte boundary on (swizzle atoms).  By an offset and not by rounding the address: a
// pointer that went through an integer is no longer known to be a shared one, and every access through it is a generic one (us,
// cold, generic / shared: attention of [1,32,2048,2048], forward with row ends 114 / 106, backward 191 / 185; layer of 2048 tokens 2122 /
// 2092, MLP of 2048 tokens 1038 / 1029).
__device__ __forceinline__ uint8_t* align_shared(uint8_t* raw) { return raw + ((0u - smem_u32(raw)) & 1023u); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {      // does not suspend
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// bounded wait; false = gave up (either the limit was hit here or another role raised abort)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 63u && *abort_flag) return false;
  }
  return false;
}
// The producer and MMA warps run their loops with all lanes and let one elected lane issue.  With `if (lane == 0)` around
// the loop nothing in it counts as warp-uniform, the descriptors of every tcgen05.mma and TMA pass through vector
// registers, and the two loops take 575-660 cycles per k-block (stamped) where the tensor pipe needs 512.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 63u) == 63u && __any_sync(0xffffffffu, *abort_flag != 0)) return false;
  }
  return false;
}
// a tile into this CTA's shared memory; the bytes are counted on the barrier at shared::cluster address `bar`,
// which in the pair form may belong to the other CTA of the pair (that is what .cta_group::2 permits)
template <bool PAIR>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  if (PAIR)
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1) : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// arrives on the barrier once the MMAs issued so far are done; pair form: on the barrier at this offset in BOTH CTAs
// (`leader`: cluster rank of the pair's first CTA)
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint64_t* bar, uint32_t leader = 0) {
  if (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)(3u << leader)) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);
  d |= (uint64_t)(lbo_bytes >> 4) << 16;
  d |= (uint64_t)(sbo_bytes >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// no swizzle, K-major: core matrices of 8 rows x 16 bytes, the two of a K = 16 slice 128 bytes apart, row groups 256
__device__ __forceinline__ uint64_t make_desc_k16(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ uint32_t k16_offset(int row, int k_half) { return (uint32_t)((row >> 3) * 256 + k_half * 128 + (row & 7) * 16); }

__device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory"); }

// round to bf16 and back: the value goes into the high half of the packed conversion, where its
// bits already are the float
__device__ __forceinline__ float bfr(float v) { return __uint_as_float(pack_bf16x2_rn(0.f, v) & 0xffff0000u); }

// ---- packed bf16x2 arithmetic.  The reference's element-wise chain works on bf16 tensors (every
// operation rounds to bf16).  For bf16 operands a packed add/sub/mul is the same thing: the fp32 product of
// two bf16 values is exact and the fp32 sum is exact unless the operands are more than 16 binades apart (then
// both forms return the larger one), so one rounding to bf16 is all that ever happens.  Two columns per
// instruction, no conversion instruction: those are the scarce resource of an epilogue that has only two
// warps per scheduler.
typedef __nv_bfloat162 bf2;
__device__ __forceinline__ bf2 as_bf2(uint32_t v) { return *reinterpret_cast<bf2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(bf2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// (the _rn forms: a multiply followed by an add must NOT be contracted into one fused operation, the
// reference rounds after each)
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) { return as_u32(__hadd2_rn(as_bf2(a), as_bf2(b))); }
__device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) { return as_u32(__hsub2_rn(as_bf2(a), as_bf2(b))); }
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) { return as_u32(__hmul2_rn(as_bf2(a), as_bf2(b))); }
constexpr uint32_t kOne2 = 0x3f803f80u;   // (1.0, 1.0)
// bf16(sigmoid(y)) of both halves; the sigmoid itself is fp32 as in the reference kernels
__device__ __forceinline__ uint32_t sigmoid2(uint32_t y) {
  const float a = bf16lo_to_f32(y), b = bf16hi_to_f32(y);
  return pack_bf16x2_rn(__fdividef(1.f, 1.f + __expf(-a)), __fdividef(1.f, 1.f + __expf(-b)));
}
// dot with an fp32 LoRA-B row in shared memory: eight packed two-wide fp32 FMAs (even and odd ranks accumulate
// side by side, one add joins them) on four 128-bit broadcast loads
__device__ __forceinline__ uint64_t pair_f32(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lora_dot_f32(const float (&xa)[16], const float* __restrict__ brow) {
  uint64_t acc = 0ull;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 b = *reinterpret_cast<const float4*>(brow + 4 * j);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(pair_f32(xa[4 * j], xa[4 * j + 1])), "l"(pair_f32(b.x, b.y)));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(pair_f32(xa[4 * j + 2], xa[4 * j + 3])), "l"(pair_f32(b.z, b.w)));
  }
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc));
  return lo + hi;
}

// LoRA terms of the GRADDOWN epilogue on the legacy tensor path (a rank-16 side product of a tcgen05 kernel)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f), "f"(0.f), "f"(0.f), "f"(0.f));
}

__device__ __forceinline__ void load_xa_row(const __nv_bfloat16* xa, int64_t row, bool valid, float (&out)[16]) {
  uint4 u = make_uint4(0u, 0u, 0u, 0u), v = u;
  if (valid && xa != nullptr) {
    u = *reinterpret_cast<const uint4*>(xa + row * 16);
    v = *reinterpret_cast<const uint4*>(xa + row * 16 + 8);
  }
  const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) { out[2 * j] = bf16lo_to_f32(w[j]); out[2 * j + 1] = bf16hi_to_f32(w[j]); }
}

// the same product with nothing staged, for the second LoRA term of a plain GEMM call (no path of the layer has one)
static __device__ __noinline__ float lora_dot_global(const LoraTerm& t, int64_t col, int64_t row, bool valid) {
  float xa[16], b[16];
  load_xa_row(t.xa, row, valid, xa);
  for (int r = 0; r < 16; ++r) b[r] = __bfloat162float(t.bt[col * t.ld_col + r * t.ld_r]);
  return lora_dot_f32(xa, b);
}

// The reference byte layout of a 32-column block: byte j carries, at bit QBIT*i, the code of
// column j + i*SLAB (SLAB = 32/EPP columns, EPP = 8/QBIT).  A block is SLAB bytes = NW words.
template <int QBIT> struct BlockGeo {
  static constexpr int EPP = 8 / QBIT, SLAB = 32 / EPP, NW = SLAB / 4;
  static constexpr uint32_t CM = (1u << QBIT) - 1u;
};

template <int QBIT>
__device__ __forceinline__ void put_code(uint32_t (&words)[BlockGeo<QBIT>::NW], int c, uint32_t code) {
  using G = BlockGeo<QBIT>;
  const int j = c % G::SLAB, i = c / G::SLAB;
  words[j >> 2] |= code << (8 * (j & 3) + QBIT * i);
}
template <int QBIT>
__device__ __forceinline__ uint32_t get_code(const uint32_t (&words)[BlockGeo<QBIT>::NW], int c) {
  using G = BlockGeo<QBIT>;
  const int j = c % G::SLAB, i = c / G::SLAB;
  return (words[j >> 2] >> (8 * (j & 3) + QBIT * i)) & G::CM;
}
template <int QBIT>
__device__ __forceinline__ void store_block_words(uint8_t* dst, const uint32_t (&w)[BlockGeo<QBIT>::NW]) {
  if constexpr (QBIT == 8) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(dst + 16) = make_uint4(w[4], w[5], w[6], w[7]);
  } else if constexpr (QBIT == 4) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
  }
}
template <int QBIT>
__device__ __forceinline__ void load_block_words(const uint8_t* src, bool valid, uint32_t (&w)[BlockGeo<QBIT>::NW]) {
#pragma unroll
  for (int i = 0; i < BlockGeo<QBIT>::NW; ++i) w[i] = 0u;
  if (!valid) return;
  if constexpr (QBIT == 8) {
    const uint4 a = *reinterpret_cast<const uint4*>(src), b = *reinterpret_cast<const uint4*>(src + 16);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  } else if constexpr (QBIT == 4) {
    const uint4 a = *reinterpret_cast<const uint4*>(src);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
  } else {
    const uint2 a = *reinterpret_cast<const uint2*>(src);
    w[0] = a.x; w[1] = a.y;
  }
}

// ------------------------------------------------------------------ epilogues (one 32-column chunk per call)
// cb = column offset of the chunk inside the tile, ncol0 = first output column of the tile.  The thread owns
// one row; columns are handled two at a time as packed bf16 pairs.
__device__ __forceinline__ void store4_pairs(__nv_bfloat16* dst, const uint32_t (&v)[4]) {
  *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
}

// Word index of 16-byte chunk c (eight columns) of a row in a [32 rows][32 columns] bf16 tile of one epilogue warp.
// The chunks of a row are permuted by the row number so that the access patterns of the epilogues
// are free of bank conflicts: 32-bit stores in the mma fragment layout (rows g, g + 8 / word t of chunk nt), 128-bit
// accesses of a lane to its own row, and 128-bit reads of eight rows x four chunks for the coalesced flush.
__device__ __forceinline__ int gd_chunk(int row, int c) { return row * 16 + ((c ^ ((row >> 1) & 3)) << 2); }

// rows [8k, 8k + 8) of the warp's tile leave as 64 contiguous bytes per row (four lanes per row)
__device__ __forceinline__ void gd_flush(const uint32_t* R, __nv_bfloat16* out, int64_t row0, int64_t M, int64_t ldo,
                                         int64_t n, int lane) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = 8 * k + (lane >> 2), c = lane & 3;
    const uint4 v = *reinterpret_cast<const uint4*>(R + gd_chunk(r, c));
    if (row0 + r < M) *reinterpret_cast<uint4*>(out + (row0 + r) * ldo + n + 8 * c) = v;
  }
}

// the opposite direction: a [32 rows][32 columns] bf16 tile as 64 contiguous bytes per row, four lanes per row
__device__ __forceinline__ void tile_fetch(const __nv_bfloat16* src, int64_t row0, int64_t M, int64_t ld, int64_t n, int lane, uint4 (&v)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = 8 * k + (lane >> 2), c = lane & 3;
    v[k] = make_uint4(0u, 0u, 0u, 0u);
    if (row0 + r < M) v[k] = *reinterpret_cast<const uint4*>(src + (row0 + r) * ld + n + 8 * c);
  }
}
__device__ __forceinline__ void tile_put(uint32_t* R, int lane, const uint4 (&v)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(R + gd_chunk(8 * k + (lane >> 2), lane & 3)) = v[k];
}

// ---- rank-16 LoRA products of the epilogues, on the legacy tensor path (side products of a tcgen05 kernel): a warp's 32
// rows x 32 columns from mma.sync fragments.  As dot products with the B rows broadcast from shared memory the same
// terms took 24-30 k cycles per 256-column tile, as long as the main loop of the next one.
struct LoraA { uint32_t f[2][4]; };      // 32 rows of xa as two 16-row A fragments
struct LoraB { uint32_t f[8]; };         // 32 columns of B^T as four 8-column B fragments
__device__ __forceinline__ void lora_load_a(const __nv_bfloat16* xa, int64_t row0, int64_t M, int lane, LoraA& a) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
    const int64_t ra = row0 + 16 * mt + g, rb = ra + 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) a.f[mt][j] = 0u;
    if (xa != nullptr) {
      if (ra < M) {
        a.f[mt][0] = *reinterpret_cast<const uint32_t*>(xa + ra * 16 + 2 * t);
        a.f[mt][2] = *reinterpret_cast<const uint32_t*>(xa + ra * 16 + 2 * t + 8);
      }
      if (rb < M) {
        a.f[mt][1] = *reinterpret_cast<const uint32_t*>(xa + rb * 16 + 2 * t);
        a.f[mt][3] = *reinterpret_cast<const uint32_t*>(xa + rb * 16 + 2 * t + 8);
      }
    }
  }
}
__device__ __forceinline__ void lora_load_b(const LoraTerm& l, int64_t n, int lane, LoraB& b) {
  const int g = lane >> 2, t = lane & 3;
  const bool fast = l.ld_r == 1 && (l.ld_col & 1) == 0 && (reinterpret_cast<uintptr_t>(l.bt) & 3) == 0;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const __nv_bfloat16* p = l.bt + (n + 8 * nt + g) * l.ld_col;
    if (fast) {
      b.f[2 * nt] = *reinterpret_cast<const uint32_t*>(p + 2 * t);
      b.f[2 * nt + 1] = *reinterpret_cast<const uint32_t*>(p + 2 * t + 8);
    } else {
      auto two = [&](int64_t r) {
        return (uint32_t)__bfloat16_as_ushort(p[r * l.ld_r]) | ((uint32_t)__bfloat16_as_ushort(p[(r + 1) * l.ld_r]) << 16);
      };
      b.f[2 * nt] = two(2 * t);
      b.f[2 * nt + 1] = two(2 * t + 8);
    }
  }
}
// the product as bf16 into the warp's tile R
__device__ __forceinline__ void lora_tile(const LoraA& a, const LoraB& b, uint32_t* R, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      float d[4];
      mma_bf16_16816(d, a.f[mt], b.f[2 * nt], b.f[2 * nt + 1]);
      // fragment: (row 16 mt + g, columns 8 nt + 2t, +1) and (row 16 mt + g + 8, same columns)
      R[gd_chunk(16 * mt + g, nt) + t] = pack_bf16x2_rn(d[0], d[1]);
      R[gd_chunk(16 * mt + g + 8, nt) + t] = pack_bf16x2_rn(d[2], d[3]);
    }
  }
}

// R1, R2: the warp's two tiles (LoRA terms in, the result out through R1)
template <int QBIT>
__device__ __forceinline__ void epi_gateup_block(const Params& p, int64_t row0, int lane, int ncol0, int cb,
                                                 const uint32_t (&g)[32], const uint32_t (&u)[32],
                                                 const LoraA& a1, const LoraA& a2, const LoraB& b1, const LoraB& b2,
                                                 const float* sR1, const float* sR2, uint32_t* R1, uint32_t* R2) {
  using G = BlockGeo<QBIT>;
  const int64_t n = (int64_t)ncol0 + cb, row = row0 + lane;
  const bool valid = row < p.M;
  lora_tile(a1, b1, R1, lane);
  lora_tile(a2, b2, R2, lane);
  __syncwarp();
  uint32_t w1[G::NW], w2[G::NW];
#pragma unroll
  for (int i = 0; i < G::NW; ++i) { w1[i] = 0u; w2[i] = 0u; }
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8) {
    const uint4 l1v = *reinterpret_cast<const uint4*>(R1 + gd_chunk(lane, c8)), l2v = *reinterpret_cast<const uint4*>(R2 + gd_chunk(lane, c8));
    const uint32_t l1[4] = {l1v.x, l1v.y, l1v.z, l1v.w}, l2[4] = {l2v.x, l2v.y, l2v.z, l2v.w};
    float r1[8], r2[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      *reinterpret_cast<float4*>(r1 + 4 * h) = *reinterpret_cast<const float4*>(sR1 + cb + 8 * c8 + 4 * h);
      *reinterpret_cast<float4*>(r2 + 4 * h) = *reinterpret_cast<const float4*>(sR2 + cb + 8 * c8 + 4 * h);
    }
    uint32_t o[4];
#pragma unroll
    for (int e2 = 0; e2 < 4; ++e2) {
      const int c = 8 * c8 + 2 * e2;
      // the frozen-weight products are bf16 tensors in the reference before anything else touches them
      const uint32_t x1 = pack_bf16x2_rn(__uint_as_float(g[c]), __uint_as_float(g[c + 1]));
      const uint32_t x2 = pack_bf16x2_rn(__uint_as_float(u[c]), __uint_as_float(u[c + 1]));
      put_code<QBIT>(w1, c, fastq_code_bits<QBIT>(bf16lo_to_f32(x1), r1[2 * e2]) & G::CM);
      put_code<QBIT>(w1, c + 1, fastq_code_bits<QBIT>(bf16hi_to_f32(x1), r1[2 * e2 + 1]) & G::CM);
      put_code<QBIT>(w2, c, fastq_code_bits<QBIT>(bf16lo_to_f32(x2), r2[2 * e2]) & G::CM);
      put_code<QBIT>(w2, c + 1, fastq_code_bits<QBIT>(bf16hi_to_f32(x2), r2[2 * e2 + 1]) & G::CM);
      const uint32_t y1 = add2(x1, l1[e2]);
      const uint32_t y1s = mul2(y1, sigmoid2(y1));
      o[e2] = mul2(y1s, add2(x2, l2[e2]));
    }
    *reinterpret_cast<uint4*>(R1 + gd_chunk(lane, c8)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  // through the warp's tile: a lane storing 16 bytes of its own row makes every store instruction touch 32 lines
  __syncwarp();
  gd_flush(R1, p.out0, row0, p.M, p.N, n, lane);
  if (valid) {
    store_block_words<QBIT>(p.q1 + (row * p.N + n) * QBIT / 8, w1);
    store_block_words<QBIT>(p.q2 + (row * p.N + n) * QBIT / 8, w2);
    if (p.dbg1 != nullptr) {
#pragma unroll
      for (int c8 = 0; c8 < 4; ++c8) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
          a[e2] = pack_bf16x2_rn(__uint_as_float(g[8 * c8 + 2 * e2]), __uint_as_float(g[8 * c8 + 2 * e2 + 1]));
          b[e2] = pack_bf16x2_rn(__uint_as_float(u[8 * c8 + 2 * e2]), __uint_as_float(u[8 * c8 + 2 * e2 + 1]));
        }
        store4_pairs(p.dbg1 + row * p.N + n + 8 * c8, a);
        store4_pairs(p.dbg2 + row * p.N + n + 8 * c8, b);
      }
    }
  }
  __syncwarp();
}

// the saved codes of columns c, c + 1 of a 32-column block as the bf16 pair (x_hat[c], x_hat[c + 1]),
// x_hat = bf16((code - half) * scale); sc2 = the two scales as a packed pair
template <int QBIT>
__device__ __forceinline__ uint32_t dequant_pair(const uint32_t (&w)[BlockGeo<QBIT>::NW], int c, uint32_t sc2) {
  const uint32_t c0 = get_code<QBIT>(w, c), c1 = get_code<QBIT>(w, c + 1);
  if constexpr (QBIT == 8) {
    // codes reach 255: through fp32 (2^23 + code), one rounding in the packed conversion
    const float f0 = (__uint_as_float(0x4B000000u | c0) - 8388736.f) * bf16lo_to_f32(sc2);
    const float f1 = (__uint_as_float(0x4B000000u | c1) - 8388736.f) * bf16hi_to_f32(sc2);
    return pack_bf16x2_rn(f0, f1);
  } else {
    // 0x4300 | code is the bf16 128 + code; minus (128 + half) is exact, the product rounds once
    constexpr uint32_t C1 = 0x4300u | (uint32_t)(1 << (QBIT - 1));
    const uint32_t pr = 0x43004300u | c0 | (c1 << 16);
    return mul2(sub2(pr, C1 | (C1 << 16)), sc2);
  }
}

// What a GRADDOWN block reads from global memory, fetched one block ahead: the packed codes of the lane's row and
// the LoRA-B fragments of the block's 32 columns for both branches.
template <int QBIT>
struct GdInputs {
  uint32_t w1[BlockGeo<QBIT>::NW], w2[BlockGeo<QBIT>::NW];
  LoraB b1, b2;
};
template <int QBIT>
__device__ __forceinline__ void gd_fetch(const Params& p, int64_t row0, int lane, int64_t n, GdInputs<QBIT>& in) {
  const int64_t row = row0 + lane;
  const bool valid = row < p.M;
  load_block_words<QBIT>(p.q1 + (row * p.N + n) * QBIT / 8, valid, in.w1);
  load_block_words<QBIT>(p.q2 + (row * p.N + n) * QBIT / 8, valid, in.w2);
  if (p.lpre1 != nullptr) return;      // kernel-uniform: the LoRA terms come from a launch that prepared them
  lora_load_b(p.l1, n, lane, in.b1);
  lora_load_b(p.l2, n, lane, in.b2);
}

// the codes alone (pair form)
template <int QBIT> struct GdCodes { uint32_t w1[BlockGeo<QBIT>::NW], w2[BlockGeo<QBIT>::NW]; };
template <int QBIT>
__device__ __forceinline__ void gd_codes(const Params& p, int64_t row, int64_t n, GdCodes<QBIT>& in) {
  const bool valid = row < p.M;
  load_block_words<QBIT>(p.q1 + (row * p.N + n) * QBIT / 8, valid, in.w1);
  load_block_words<QBIT>(p.q2 + (row * p.N + n) * QBIT / 8, valid, in.w2);
}

// One block of 32 rows x 32 columns of the GRADDOWN epilogue, a whole warp at a time (lane = row for the
// accumulator and the element-wise chain).  The LoRA terms of the two branches are rank-16 products on the legacy
// tensor path: fragments -> bf16 pairs -> the warp's two shared-memory tiles, from which every lane reads its own
// row.  The same tiles then collect the results so that they leave as coalesced 64-byte row segments: a lane
// storing 16 bytes of its own row would make every store instruction touch 32 lines, which throttled the
// load/store unit and slowed the TMA loads of the main loop.
template <int QBIT>
__device__ __forceinline__ void epi_graddown_block(const Params& p, int64_t row0, int lane, int ncol0, int cb,
                                                   const uint32_t (&acc)[32], const GdInputs<QBIT>& in,
                                                   const LoraA& a1, const LoraA& a2,
                                                   uint32_t* R1, uint32_t* R2,
                                                   const uint32_t* sS1, const uint32_t* sS2) {
  const int64_t n = (int64_t)ncol0 + cb;
  const int64_t row = row0 + lane;
  const bool valid = row < p.M;
  const bool pre = p.lpre1 != nullptr;      // kernel-uniform
  if (!pre) {
    lora_tile(a1, in.b1, R1, lane);
    lora_tile(a2, in.b2, R2, lane);
    __syncwarp();
  }
  uint32_t gu_all[16];
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8) {
    uint32_t o[4], gg[4];
    // the LoRA terms of the lane's row: from the warp's tiles, or from a launch that prepared them
    uint4 pl1, pl2;
    if (pre) {
      pl1 = make_uint4(0u, 0u, 0u, 0u); pl2 = pl1;
      if (valid) {
        pl1 = *reinterpret_cast<const uint4*>(p.lpre1 + row * p.ld_pre + n + 8 * c8);
        pl2 = *reinterpret_cast<const uint4*>(p.lpre2 + row * p.ld_pre + n + 8 * c8);
      }
    } else {
      pl1 = *reinterpret_cast<const uint4*>(R1 + gd_chunk(lane, c8));
      pl2 = *reinterpret_cast<const uint4*>(R2 + gd_chunk(lane, c8));
    }
    const uint32_t pw1[4] = {pl1.x, pl1.y, pl1.z, pl1.w}, pw2[4] = {pl2.x, pl2.y, pl2.z, pl2.w};
#pragma unroll
    for (int e2 = 0; e2 < 4; ++e2) {
      const int c = 8 * c8 + 2 * e2, tc = cb + c;
      // the LoRA part of grad_down arrived as an extra K block
      const uint32_t gd = pack_bf16x2_rn(__uint_as_float(acc[c]), __uint_as_float(acc[c + 1]));
      const uint32_t x1 = dequant_pair<QBIT>(in.w1, c, sS1[tc >> 1]);
      const uint32_t x2 = dequant_pair<QBIT>(in.w2, c, sS2[tc >> 1]);
      const uint32_t y1 = add2(x1, pw1[e2]), sig = sigmoid2(y1), y1s = mul2(y1, sig), y2 = add2(x2, pw2[e2]);
      o[e2] = mul2(y1s, y2);
      gu_all[4 * c8 + e2] = mul2(gd, y1s);
      const uint32_t inner = add2(kOne2, mul2(y1, sub2(kOne2, sig)));
      gg[e2] = mul2(mul2(gd, y2), mul2(sig, inner));
    }
    // chunk c8 of the lane's own row is dead now: the results take its place
    *reinterpret_cast<uint4*>(R1 + gd_chunk(lane, c8)) = make_uint4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint4*>(R2 + gd_chunk(lane, c8)) = make_uint4(gg[0], gg[1], gg[2], gg[3]);
  }
  __syncwarp();
  gd_flush(R1, p.out0, row0, p.M, p.N, n, lane);
  gd_flush(R2, p.out1, row0, p.M, p.N, n, lane);
  __syncwarp();
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8)
    *reinterpret_cast<uint4*>(R1 + gd_chunk(lane, c8)) = make_uint4(gu_all[4 * c8], gu_all[4 * c8 + 1], gu_all[4 * c8 + 2], gu_all[4 * c8 + 3]);
  __syncwarp();
  gd_flush(R1, p.out2, row0, p.M, p.N, n, lane);
  __syncwarp();     // the tiles are rewritten by the next block
}

// `res`: the block's residual as tile_fetch left it; L, R: the warp's tiles for the LoRA term and for
// residual and result, which travel through it so
// that global accesses are whole 64-byte row segments
template <int QBIT>
__device__ __forceinline__ void epi_store_block(const StoreView& v, int64_t row0, int lane, int64_t M, int cb,
                                                const uint32_t (&acc)[32], const LoraA& a0, const LoraB& b0, const float* sR,
                                                const uint4 (&res)[4], uint32_t* L, uint32_t* R) {
  using G = BlockGeo<QBIT>;
  const int64_t n = (int64_t)v.n0 + cb, row = row0 + lane;
  const bool valid = row < M;
  const bool has0 = v.l0.bt != nullptr, has1 = v.l1.bt != nullptr;
  const bool has_res = v.residual != nullptr;
  const bool save = v.q != nullptr;
  uint32_t w1[G::NW];
#pragma unroll
  for (int i = 0; i < G::NW; ++i) w1[i] = 0u;
  if (has0) lora_tile(a0, b0, L, lane);
  if (has_res) tile_put(R, lane, res);
  if (has0 || has_res) __syncwarp();
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8) {
    uint4 rq = make_uint4(0u, 0u, 0u, 0u);
    if (has_res) rq = *reinterpret_cast<const uint4*>(R + gd_chunk(lane, c8));
    const uint32_t r[4] = {rq.x, rq.y, rq.z, rq.w};
    uint4 lq = make_uint4(0u, 0u, 0u, 0u);
    if (has0) lq = *reinterpret_cast<const uint4*>(L + gd_chunk(lane, c8));
    const uint32_t l[4] = {lq.x, lq.y, lq.z, lq.w};
    float rs[8];
    if (save) {
#pragma unroll
      for (int h = 0; h < 2; ++h) *reinterpret_cast<float4*>(rs + 4 * h) = *reinterpret_cast<const float4*>(sR + cb + 8 * c8 + 4 * h);
    }
    uint32_t o[4], m[4];
#pragma unroll
    for (int e2 = 0; e2 < 4; ++e2) {
      const int c = 8 * c8 + 2 * e2, tc = cb + c;
      uint32_t y = pack_bf16x2_rn(__uint_as_float(acc[c]), __uint_as_float(acc[c + 1]));
      m[e2] = y;
      if (save) {
        put_code<QBIT>(w1, c, fastq_code_bits<QBIT>(bf16lo_to_f32(y), rs[2 * e2]) & G::CM);
        put_code<QBIT>(w1, c + 1, fastq_code_bits<QBIT>(bf16hi_to_f32(y), rs[2 * e2 + 1]) & G::CM);
      }
      if (has0) y = add2(y, l[e2]);
      if (has1) y = add2(y, pack_bf16x2_rn(lora_dot_global(v.l1, v.n0 + tc, row, valid), lora_dot_global(v.l1, v.n0 + tc + 1, row, valid)));
      if (has_res) y = add2(y, r[e2]);
      o[e2] = y;
    }
    *reinterpret_cast<uint4*>(R + gd_chunk(lane, c8)) = make_uint4(o[0], o[1], o[2], o[3]);
    if (valid && v.main != nullptr) store4_pairs(v.main + row * v.ld + n + 8 * c8, m);
  }
  __syncwarp();
  gd_flush(R, v.out, row0, M, v.ld, n, lane);
  __syncwarp();
  if (save && valid) store_block_words<QBIT>(v.q + (row * v.ld + n) * QBIT / 8, w1);
}

// ------------------------------------------------------------------ epilogues of the pair form
// The rank-16 LoRA terms come from tcgen05 as well: once the warps of both CTAs have the main branch of a tile in registers
// (as bf16 pairs), its tensor-memory columns are free and take bf16 xa B^T as one K = 16 product each.  From mma.sync
// fragments the same terms queued behind the busy tensor pipe: the epilogue of the gate/up product took 38 k cycles where
// the main loop of the next tile takes 34 k (2048 tokens, Llama-2-7B: 293 us; without those instructions 237).
struct LoraStage { uint8_t *a1, *a2, *b1, *b2; };      // [128][16] and [columns / 2][16] operands, k16_offset layout

// 16-byte chunks of operand rows, by the 256 epilogue threads (et)
__device__ __forceinline__ void stage_lora_a(uint8_t* dst, const __nv_bfloat16* xa, int64_t m0, int64_t M, int et) {
  const int row = et >> 1, kh = et & 1;
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (m0 + row < M) v = *reinterpret_cast<const uint4*>(xa + (m0 + row) * 16 + 8 * kh);
  *reinterpret_cast<uint4*>(dst + k16_offset(row, kh)) = v;
}
__device__ __forceinline__ void stage_lora_b(uint8_t* dst, const LoraTerm& l, int64_t n, int rows, int et) {
  const int row = et >> 1, kh = et & 1;
  if (row >= rows) return;
  const __nv_bfloat16* p = l.bt + (n + row) * l.ld_col + 8 * kh * l.ld_r;
  uint4 v;
  if (l.ld_r == 1 && (l.ld_col & 7) == 0 && (reinterpret_cast<uintptr_t>(l.bt) & 15) == 0) {
    v = *reinterpret_cast<const uint4*>(p);
  } else {
    auto two = [&](int r) { return (uint32_t)__bfloat16_as_ushort(p[r * l.ld_r]) | ((uint32_t)__bfloat16_as_ushort(p[(r + 1) * l.ld_r]) << 16); };
    v = make_uint4(two(0), two(2), two(4), two(6));
  }
  *reinterpret_cast<uint4*>(dst + k16_offset(row, kh)) = v;
}

// 32 accumulator columns of the lane's row as 16 bf16 pairs
__device__ __forceinline__ void tc_ld_pairs(uint32_t taddr, uint32_t (&x)[16]) {
  uint32_t v[32];
  tc_ld32(taddr, v);
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = pack_bf16x2_rn(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
}
// the block's codes; r: its quantizer constants in shared memory
template <int QBIT>
__device__ __forceinline__ void pack_codes(const uint32_t (&x)[16], const float* r, uint32_t (&w)[BlockGeo<QBIT>::NW]) {
  using G = BlockGeo<QBIT>;
#pragma unroll
  for (int i = 0; i < G::NW; ++i) w[i] = 0u;
#pragma unroll
  for (int c = 0; c < 32; c += 4) {
    const float4 k = *reinterpret_cast<const float4*>(r + c);
    put_code<QBIT>(w, c, fastq_code_bits<QBIT>(bf16lo_to_f32(x[c / 2]), k.x) & G::CM);
    put_code<QBIT>(w, c + 1, fastq_code_bits<QBIT>(bf16hi_to_f32(x[c / 2]), k.y) & G::CM);
    put_code<QBIT>(w, c + 2, fastq_code_bits<QBIT>(bf16lo_to_f32(x[c / 2 + 1]), k.z) & G::CM);
    put_code<QBIT>(w, c + 3, fastq_code_bits<QBIT>(bf16hi_to_f32(x[c / 2 + 1]), k.w) & G::CM);
  }
}
// a lane's 16 pairs through the warp's tile: out as whole 64-byte row segments
__device__ __forceinline__ void flush_pairs(const uint32_t (&o)[16], uint32_t* R, __nv_bfloat16* out, int64_t row0, int64_t M, int64_t ldo, int64_t n,
                                            int lane) {
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8)
    *reinterpret_cast<uint4*>(R + gd_chunk(lane, c8)) = make_uint4(o[4 * c8], o[4 * c8 + 1], o[4 * c8 + 2], o[4 * c8 + 3]);
  __syncwarp();
  gd_flush(R, out, row0, M, ldo, n, lane);
  __syncwarp();
}
__device__ __forceinline__ void store_pairs(const uint32_t (&o)[16], __nv_bfloat16* dst) {
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8) *reinterpret_cast<uint4*>(dst + 8 * c8) = make_uint4(o[4 * c8], o[4 * c8 + 1], o[4 * c8 + 2], o[4 * c8 + 3]);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode() {
  // the encoder is a driver function: a thread whose first CUDA work is this call has no context current yet (the
  // runtime binds the device's primary context, once per thread)
  static thread_local bool bound = false;
  if (!bound) {
    int dev = 0;
    bound = cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess;
  }
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// row-major bf16 matrix [rows, cols] (cols contiguous), box = 64 columns x box_rows rows, 128-byte swizzle
inline bool make_map(CUtensorMap* m, const void* ptr, int64_t rows, int64_t cols, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1u, 1u};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// the matrices behind the maps: row-major, p == nullptr repeats entry 0
struct Matrix { const void* p; int64_t rows, cols; };
struct Operands { Matrix a[4], b[4]; };
inline bool make_maps(Maps* m, const Operands& o, bool b_mn, int a_rows, int b_rows, bool narrow) {
  for (int i = 0; i < 4; ++i) {
    if (o.a[i].p == nullptr) m->a[i] = m->a[0];
    else if (!make_map(&m->a[i], o.a[i].p, o.a[i].rows, o.a[i].cols, a_rows)) return false;
    if (o.b[i].p == nullptr) { m->b[i] = m->b[0]; m->n[i] = m->n[0]; continue; }
    if (!make_map(&m->b[i], o.b[i].p, o.b[i].rows, o.b[i].cols, b_mn ? 64 : b_rows)) return false;
    m->n[i] = m->b[i];
    if (narrow && !b_mn && !make_map(&m->n[i], o.b[i].p, o.b[i].rows, o.b[i].cols, 64)) return false;
  }
  return true;
}

}  // namespace tc
}  // namespace hyc
