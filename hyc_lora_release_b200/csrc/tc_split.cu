// The GEMMs of the layer for few tokens: one 128 x 128 tile per cluster of S = 1, 2 or 4 CTAs, each CTA contracting
// one S-th of K; the partial accumulators meet in distributed shared memory and every CTA finishes 1/S of the tile's
// columns with the same epilogues as the persistent kernel (mlp_tcgen05.cu).
//
// Why: below about a thousand tokens a 256 x 256 tile per CTA pair leaves most of the chip idle ([128, 4096] x
// [4096, 4096]: 16 tiles on 74 pairs) while the product is bound by streaming the weights from HBM.  Here every SM
// streams its own slice of the weight with two CTAs of three 32 KB stages (or one of six) in flight; the A tile comes
// from L2.  With 129 tokens and more the tile belongs to a CTA pair (M 256, tcgen05 cta_group::2, each CTA loading half
// of the B block), which cuts what an SM pulls out of L2 per k-block from 32 to 24 KB; a cluster is then 2 S CTAs.
// The reduction order is fixed (rank 0, 1, ...), so results do not depend on the run.
//
// FOUR: frozen weights that are 4-bit codes.  Up to 128 rows every element of a weight is read by one CTA alone, so that decoding it there
// costs no more than decoding it once, and what a launch of its own would write and the product read back, 2 + 2 bytes per element, is not
// moved at all.  Eight warps write the B blocks where TMA would have put them, two k-blocks at a time, a thread the 64 elements of a
// 128-byte row (32 bytes of codes under one scale): the sixteen values that a scale makes of the table as byte planes in registers, then
// byte permutes (3.7 instructions per element).  Bound by instructions (issue slots 0.37, two and a half warps per scheduler) and by the
// requests for codes and scales, 32 and 4 bytes per thread from rows of their own: 0.65 us per k-block, 0.59 without the arithmetic, 0.42
// without the requests.  The launch bound (two CTAs of 320 threads per SM, which only gate and up of a wide MLP fill) leaves 96 registers per
// thread: the store forms spill 192 bytes per thread, gate/up about 400, grad_down up to 36.  The products of a layer of 128 tokens that take
// codes, us: 395 as de-quantizing launches and products, 328 so; the layer step 577 -> 507 (its host work takes about as long).  More codes in
// flight (cp.async, eight slots), sixteen warps, and addresses carried from block to block gave nothing or cost some.  Which products: four_pays().
#include "tc_split.cuh"

namespace hyc {
namespace tc {

constexpr int SBN = 128;                          // accumulator columns per tile
constexpr int S_PIPE_BYTES = 98304;               // pipeline memory of a CTA that shares its SM (twice that if it does not)
constexpr int S_MAX_STAGES = 8;
constexpr int S_EPI_BYTES = 1024;                 // per-column constants
constexpr int S_THREADS = 64 + 128;
constexpr int S_PART_BYTES = SBN * BM * 4;        // the CTA's accumulators as [column][row], over the drained stages
static_assert(S_PART_BYTES + 4 * 4096 <= S_PIPE_BYTES, "partials and the epilogue's tiles fit in the drained pipeline");
constexpr int split_smem_bytes(int pipe) { return 1024 + pipe + S_EPI_BYTES + 256; }

__device__ __forceinline__ void s_epi_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// 32 accumulator columns from `col` of the thread's row: this CTA's tensor memory, or the sum over the cluster
// (its CTAs that hold the same rows: ranks first, first + step, ...)
__device__ __forceinline__ void gather32(int split, int first, int step, uint32_t t_lane, uint32_t part, int col, int r,
                                         uint32_t (&acc)[32]) {
  if (split == 1) {
    tc_ld32(t_lane + (uint32_t)col, acc);
    return;
  }
  float f[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) f[c] = 0.f;
  for (int s = 0; s < split; ++s) {
    uint32_t base;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base) : "r"(part + (uint32_t)(col * BM + r) * 4u), "r"(first + s * step));
#pragma unroll
    for (int c = 0; c < 32; ++c) f[c] += ld_cluster_f32(base + (uint32_t)(c * BM * 4));
  }
#pragma unroll
  for (int c = 0; c < 32; ++c) acc[c] = __float_as_uint(f[c]);
}

// ---- 4-bit weights
constexpr int S_FOUR_WARPS = 8, S_FOUR_AT = 512;      // decoding warps; where the tables lie in the epilogue's constants
static_assert(S_FOUR_AT + 4 * 64 <= S_EPI_BYTES, "the tables fit behind the constants");
// 64 elements on their way: their codes and what makes their scale
struct FourUnit {
  uint32_t w[8];
  float s, c;                               // absmax; two-level: the second-level factor and the table value
  uint32_t q;                               // two-level: the code
  int which;                                // weight, -1: nothing to decode
};
__device__ __forceinline__ void four_fetch(const FourView& v, int which, int64_t e, FourUnit& u) {
  asm volatile("ld.global.L2::128B.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(u.w[0]), "=r"(u.w[1]), "=r"(u.w[2]), "=r"(u.w[3]), "=r"(u.w[4]), "=r"(u.w[5]), "=r"(u.w[6]), "=r"(u.w[7]) : "l"(v.packed + e / 2));
  const int64_t blk = e >> v.shift;
  u.which = which;
  u.q = 0u;
  if (v.absmax) {
    u.s = v.absmax[blk];
  } else {
    u.q = v.absmax_q[blk];
    u.s = v.absmax2[blk >> v.shift2];
  }
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {      // bit 3 of a selector: the byte's sign, eight times
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// to the 128-byte row at `row`, whose 16-byte chunks lie permuted by `swz`
__device__ __forceinline__ void four_decode(const FourUnit& u, float s, const float* code, uint8_t* row, int swz) {
  uint32_t lo[4], hi[4];                    // the low and the high bytes of the sixteen values
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 c = *reinterpret_cast<const float4*>(code + 4 * i);
    const uint32_t a = pack_bf16x2_rn(__fmul_rn(c.x, s), __fmul_rn(c.y, s)), b = pack_bf16x2_rn(__fmul_rn(c.z, s), __fmul_rn(c.w, s));
    lo[i] = prmt(a, b, 0x6420u);
    hi[i] = prmt(a, b, 0x7531u);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t sel = u.w[c] & 0x77777777u, z = u.w[c] << 4;
    uint32_t o[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // four codes, the low nibble of a byte before the high one; which of them are in the upper half of the table
      const uint32_t k = h ? sel >> 16 : sel, up = prmt(u.w[c], z, h ? 0xbfaeu : 0x9d8cu);
      const uint32_t l = (prmt(lo[0], lo[1], k) & ~up) | (prmt(lo[2], lo[3], k) & up);
      const uint32_t m = (prmt(hi[0], hi[1], k) & ~up) | (prmt(hi[2], hi[3], k) & up);
      o[2 * h] = prmt(l, m, 0x4051u);       // (the high nibble is the first element)
      o[2 * h + 1] = prmt(l, m, 0x6273u);
    }
    *reinterpret_cast<uint4*>(row + ((c ^ swz) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int EPI, int QBIT, bool B_MN, bool PAIR, bool FOUR>
__global__ void __launch_bounds__(FOUR ? 64 + 32 * S_FOUR_WARPS : S_THREADS, 2)
split_gemm_kernel(const __grid_constant__ Maps maps, const Params p, int split, int stages, int a_bytes, const __grid_constant__ FourWeights four) {
  static_assert(EPI == EPI_STORE || (EPI == EPI_GATEUP && !PAIR && !B_MN) || (EPI == EPI_GRADDOWN && FOUR && B_MN), "the forms that are launched");
  static_assert(!(FOUR && PAIR), "a pair would decode everything twice");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  constexpr int TILE_M = PAIR ? 2 * BM : BM;
  constexpr int B_BYTES = (PAIR ? SBN / 2 : SBN) * BK * 2;        // this CTA's part of the B block
  const int stage_bytes = a_bytes + B_BYTES;
  uint8_t* epi = smem + (stages * stage_bytes + 1023) / 1024 * 1024;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi + S_EPI_BYTES);
  uint64_t *full = bars, *empty = bars + S_MAX_STAGES, *acc_full = bars + 2 * S_MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S_MAX_STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int crank = PAIR || split > 1 ? (int)cluster_ctarank() : 0;
  const int half = PAIR ? crank & 1 : 0, rank = PAIR ? crank >> 1 : crank;      // which rows of the tile, which slice of K
  const uint32_t leader = (uint32_t)(crank & ~1);                               // PAIR: the CTA that issues the pair's MMAs
  constexpr int TILE_N = EPI == EPI_GATEUP ? SBN / 2 : SBN;
  constexpr int UNITS = TILE_N / 32;
  const int tiles_m = (p.M + TILE_M - 1) / TILE_M;
  const int tile = (int)blockIdx.x / (PAIR ? 2 * split : split);
  const int m0 = (tile % tiles_m) * TILE_M + half * BM, nt = (tile / tiles_m) * TILE_N;
  const int kb1 = p.K1 / BK, kb2 = (p.K1 + p.K2) / BK, kb3 = (p.K1 + p.K2 + p.K3) / BK, kb_total = kb3 + p.K4 / BK;
  const int kb_lo = (int)((int64_t)kb_total * rank / split), kb_hi = (int)((int64_t)kb_total * (rank + 1) / split);
  const StoreView sv = store_view(p, nt);

  if (threadIdx.x == 0) {
    // (FOUR: a B block is there when the four warps that decode it have arrived)
    for (int s = 0; s < stages; ++s) { mbar_init(&full[s], FOUR ? 1 + S_FOUR_WARPS / 2 : 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();      // before tensor memory is taken: see launch_pdl
  if (FOUR && threadIdx.x >= 64 && threadIdx.x < 64 + 64) {
    const int i = (int)threadIdx.x - 64;
    if (four.w[i >> 4].packed != nullptr) reinterpret_cast<float*>(epi + S_FOUR_AT)[i] = four.w[i >> 4].code16[i & 15];
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(SBN) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(SBN) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the peer's barriers exist before anything is signalled there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int et = (int)threadIdx.x - 64, quad = warp & 3;
  const int64_t row0 = (int64_t)m0 + quad * 32;
  const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
  float* part = reinterpret_cast<float*>(smem);
  float* sV = reinterpret_cast<float*>(epi);                       // quantizer constants (GATEUP: second vector at sV + 64)
  const int per = UNITS / split, first = rank * per;               // the 32-column blocks this CTA finishes
  LoraA a1, a2;
  LoraB b1, b2;
  uint4 res[4];
  bool ok = true;

  if (warp == 0) {
    {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1u, abort_flag)) {
          if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_PRODUCER); }
          break;
        }
        const int seg = kb < kb1 ? 0 : (kb < kb2 ? 1 : (kb < kb3 ? 2 : 3));
        const int wsel = EPI == EPI_STORE && sv.group > 0 ? sv.group : seg;
        const CUtensorMap *ma = &maps.a[seg], *mb = &maps.b[wsel];
        const int k0 = (kb - (seg == 0 ? 0 : (seg == 1 ? kb1 : (seg == 2 ? kb2 : kb3)))) * BK;
        const int n0 = EPI == EPI_STORE ? sv.n0 : nt;
        const uint32_t sa = smem_u32(smem + stage * stage_bytes), sb = sa + (uint32_t)a_bytes;
        const uint32_t fbar = PAIR ? map_to_cta(&full[stage], leader) : smem_u32(&full[stage]);
        if (elect_one()) {
        const bool decoded = FOUR && four.w[wsel].packed != nullptr;
        if (half == 0) mbar_expect_tx(&full[stage], (uint32_t)((PAIR ? 2 : 1) * (decoded ? a_bytes : stage_bytes)));      // the leader counts both CTAs' bytes
        if (decoded) {
        } else if (EPI == EPI_GATEUP) {
          tma_load_2d<PAIR>(sb, &maps.b[0], fbar, k0, n0);
          tma_load_2d<PAIR>(sb + 8192, &maps.b[1], fbar, k0, n0);
        } else if (B_MN) {
          tma_load_2d<PAIR>(sb, mb, fbar, n0 + 64 * half, k0);
          if (!PAIR) tma_load_2d<PAIR>(sb + 8192, mb, fbar, n0 + 64, k0);
        } else {
          tma_load_2d<PAIR>(sb, mb, fbar, k0, n0 + 64 * half);
        }
        tma_load_2d<PAIR>(sa, ma, fbar, k0, m0);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (half == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((B_MN ? 1u : 0u) << 16) | ((uint32_t)(SBN >> 3) << 17) |
                             ((uint32_t)(TILE_M >> 4) << 24);
      int stage = 0;
      uint32_t phase = 0;
      bool fine = true;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_warp(&full[stage], phase, abort_flag)) {
          if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_MMA); }
          fine = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * stage_bytes), sb = sa + (uint32_t)a_bytes;
        const uint64_t adesc = make_desc(sa, 16, 1024);
        const uint64_t bdesc = B_MN ? make_desc(sb, 64 * 128, 1024) : make_desc(sb, 16, 1024);
        if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
          tc_mma<PAIR>(tmem_base, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(B_MN ? kk * 128 : kk * 2), idesc,
                        (kb > kb_lo || kk > 0) ? 1u : 0u);
        tc_commit<PAIR>(&empty[stage], leader);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
      if (fine && elect_one()) tc_commit<PAIR>(acc_full, leader);
    }
    __syncwarp();
  } else {
    if constexpr (FOUR) {
      // warps 2..5 decode the even k-blocks of this CTA's share, warps 6..9 the odd ones; codes and scales are two blocks of theirs ahead
      const int group = (warp - 2) >> 2, i = ((int)threadIdx.x - 64) & 127;
      auto fetch = [&](int kb, FourUnit& u) {
        u.which = -1;
        if (kb >= kb_hi) return;
        const int seg = kb < kb1 ? 0 : (kb < kb2 ? 1 : (kb < kb3 ? 2 : 3));
        const int k0 = (kb - (seg == 0 ? 0 : (seg == 1 ? kb1 : (seg == 2 ? kb2 : kb3)))) * BK;
        const int which = EPI == EPI_GATEUP ? i >> 6 : (EPI == EPI_STORE && sv.group > 0 ? sv.group : seg);
        const FourView& v = four.w[which];
        if (v.packed == nullptr) return;      // (TMA brings it)
        const int n0 = EPI == EPI_STORE ? sv.n0 : nt;
        if (B_MN) four_fetch(v, which, (int64_t)(k0 + (i >> 1)) * v.ld + n0 + 64 * (i & 1), u);
        else four_fetch(v, which, (int64_t)(n0 + (EPI == EPI_GATEUP ? i & 63 : i)) * v.ld + k0, u);
      };
      auto table_value = [&](FourUnit& u) {
        if (u.which >= 0 && four.w[u.which].absmax == nullptr) u.c = __ldg(four.w[u.which].code256 + u.q);
      };
      const float* code = reinterpret_cast<const float*>(epi + S_FOUR_AT);
      const uint32_t row_at = B_MN ? (uint32_t)((i & 1) * 8192 + (i >> 1) * 128) : (uint32_t)(i * 128);
      const int swz = B_MN ? (i >> 1) & 7 : i & 7;
      int stage = group;
      uint32_t phase = 0;
      FourUnit n1, n2;
      fetch(kb_lo + group, n1);
      table_value(n1);
      fetch(kb_lo + group + 2, n2);
      for (int kb = kb_lo + group; kb < kb_hi; kb += 2) {
        const FourUnit u = n1;
        n1 = n2;
        table_value(n1);
        fetch(kb + 4, n2);
        if (!mbar_wait_warp(&empty[stage], phase ^ 1u, abort_flag)) {
          if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_PRODUCER); }
          break;
        }
        if (u.which >= 0) {
          const FourView& v = four.w[u.which];
          const float s = v.absmax ? u.s : __fadd_rn(__fmul_rn(u.c, u.s), v.offset);
          four_decode(u, s, code + 16 * u.which, smem + stage * stage_bytes + a_bytes + row_at, swz);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[stage]);
        stage += 2;
        if (stage >= stages) { stage -= stages; phase ^= 1u; }
      }
    }
    if (!FOUR || warp < 6) {
    // what the epilogue needs besides the accumulators is fetched while the main loop runs
    if (EPI == EPI_GRADDOWN) {
      reinterpret_cast<__nv_bfloat16*>(sV)[et] = p.s1[nt + et];
      reinterpret_cast<__nv_bfloat16*>(sV)[SBN + et] = p.s2[nt + et];
      lora_load_a(p.l1.xa, row0, p.M, lane, a1);
      lora_load_a(p.l2.xa, row0, p.M, lane, a2);
    } else if (EPI == EPI_STORE) {
      if (sv.q != nullptr) sV[et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(sv.s[sv.n0 + et])));
      if (sv.l0.bt != nullptr) {
        lora_load_a(sv.l0.xa, row0, p.M, lane, a1);
        lora_load_b(sv.l0, (int64_t)sv.n0 + 32 * first, lane, b1);
      }
      if (sv.residual != nullptr) tile_fetch(sv.residual, row0, p.M, sv.ld, (int64_t)sv.n0 + 32 * first, lane, res);
    } else {
      if (et < TILE_N) {
        sV[et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(p.s1[nt + et])));
        sV[64 + et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(p.s2[nt + et])));
      }
      lora_load_a(p.l0.xa, row0, p.M, lane, a1);
      lora_load_a(p.l1.xa, row0, p.M, lane, a2);
      lora_load_b(p.l0, (int64_t)nt + 32 * first, lane, b1);
      lora_load_b(p.l1, (int64_t)nt + 32 * first, lane, b2);
    }
    s_epi_sync();
    ok = mbar_wait(acc_full, 0, abort_flag);
    if (!ok && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_EPILOGUE); }
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    if (ok && split > 1) {
      // the stages are drained (the accumulators are complete): they hold the partial sums now
#pragma unroll 1
      for (int c0 = 0; c0 < SBN; c0 += 32) {
        uint32_t v[32];
        tc_ld32(t_lane + (uint32_t)c0, v);
#pragma unroll
        for (int c = 0; c < 32; ++c) part[(c0 + c) * BM + quad * 32 + lane] = __uint_as_float(v[c]);
      }
    }
    }
  }
  // every CTA of the cluster has its partial sums in place (or has given up: the status word says so)
  if (split > 1) cluster_sync_all();

  if (warp >= 2 && warp < 6 && ok) {
    const uint32_t part_addr = smem_u32(part);
    const int r = quad * 32 + lane;
    // behind the partial sums
    uint32_t *R1 = reinterpret_cast<uint32_t*>(smem + S_PART_BYTES) + (warp - 2) * 1024, *R2 = R1 + 512;
#pragma unroll 1
    for (int u = first; u < first + per; ++u) {
      const int cb = 32 * u;
      const bool more = u + 1 < first + per;
      uint32_t acc[32];
      if (EPI == EPI_GATEUP) {
        uint32_t up[32];
        const LoraB n1 = b1, n2 = b2;
        if (more) {
          lora_load_b(p.l0, (int64_t)nt + cb + 32, lane, b1);
          lora_load_b(p.l1, (int64_t)nt + cb + 32, lane, b2);
        }
        gather32(split, half, PAIR ? 2 : 1, t_lane, part_addr, cb, r, acc);
        gather32(split, half, PAIR ? 2 : 1, t_lane, part_addr, TILE_N + cb, r, up);
        epi_gateup_block<QBIT>(p, row0, lane, nt, cb, acc, up, a1, a2, n1, n2, sV, sV + 64, R1, R2);
      } else if constexpr (EPI == EPI_GRADDOWN) {
        GdInputs<QBIT> in;
        gd_fetch<QBIT>(p, row0, lane, (int64_t)nt + cb, in);
        gather32(split, half, 1, t_lane, part_addr, cb, r, acc);
        epi_graddown_block<QBIT>(p, row0, lane, nt, cb, acc, in, a1, a2, R1, R2, reinterpret_cast<const uint32_t*>(sV),
                                 reinterpret_cast<const uint32_t*>(sV) + SBN / 2);
      } else {
        const uint4 now[4] = {res[0], res[1], res[2], res[3]};
        const LoraB n1 = b1;
        if (more && sv.residual != nullptr) tile_fetch(sv.residual, row0, p.M, sv.ld, (int64_t)sv.n0 + cb + 32, lane, res);
        if (more && sv.l0.bt != nullptr) lora_load_b(sv.l0, (int64_t)sv.n0 + cb + 32, lane, b1);
        gather32(split, half, PAIR ? 2 : 1, t_lane, part_addr, cb, r, acc);
        epi_store_block<QBIT>(sv, row0, lane, p.M, cb, acc, a1, n1, sV, now, R1, R2);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (PAIR || split > 1) cluster_sync_all();      // nobody leaves while a peer may still read its partial sums
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SBN) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SBN) : "memory");
  }
}

template <int EPI, int QBIT, bool B_MN, bool PAIR, bool FOUR = false>
static int launch_one(int split, const Operands& ops, const Params& p, cudaStream_t st, const FourWeights& four = {}) {
  auto kern = split_gemm_kernel<EPI, QBIT, B_MN, PAIR, FOUR>;
  static bool attr[64] = {false};
  const int slot = current_device_slot();
  if (slot < 0 || !attr[slot]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, split_smem_bytes(2 * S_PIPE_BYTES)) != cudaSuccess) {
      hyc_set_last_cuda_error((int)cudaGetLastError());
      return HYC_ERR_LAUNCH;
    }
    if (slot >= 0) attr[slot] = true;
  }
  constexpr int TILE_N = EPI == EPI_GATEUP ? SBN / 2 : SBN, TILE_M = PAIR ? 2 * BM : BM;
  const int cluster = (PAIR ? 2 : 1) * split;
  const int ctas = ((p.M + TILE_M - 1) / TILE_M) * (p.N / TILE_N) * cluster;
  const int pipe = ctas <= num_sms() ? 2 * S_PIPE_BYTES : S_PIPE_BYTES;       // one CTA per SM, or room for two
  const int a_bytes = (p.M <= 64 ? 64 : BM) * BK * 2;
  const int stage_bytes = a_bytes + (PAIR ? SBN / 2 : SBN) * BK * 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(FOUR ? 64 + 32 * S_FOUR_WARPS : S_THREADS);
  cfg.dynamicSmemBytes = split_smem_bytes(pipe);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  int stages = pipe / stage_bytes;
  if (stages > S_MAX_STAGES) stages = S_MAX_STAGES;
  Maps maps = {};      // (FOUR: some weights have none)
  if (!make_maps(&maps, ops, B_MN, a_bytes / (BK * 2), EPI == EPI_GATEUP || PAIR ? 64 : 128, false)) return HYC_ERR_UNSUPPORTED;
  if (cudaLaunchKernelEx(&cfg, kern, maps, p, split, stages, a_bytes, four) != cudaSuccess) {
    hyc_set_last_cuda_error((int)cudaGetLastError());
    return HYC_ERR_LAUNCH;
  }
  return HYC_OK;
}

// (only the forms that choose_split picks: products with codes in their epilogue are never split, so never paired)
int launch_split(int epi, int q_bit, bool b_mn, const SplitPlan& plan, const Operands& ops, const Params& p, cudaStream_t st) {
  if (epi == EPI_GATEUP) {
    if (q_bit == 2) return launch_one<EPI_GATEUP, 2, false, false>(plan.split, ops, p, st);
    if (q_bit == 8) return launch_one<EPI_GATEUP, 8, false, false>(plan.split, ops, p, st);
    return launch_one<EPI_GATEUP, 4, false, false>(plan.split, ops, p, st);
  }
  if (b_mn) {
    if (plan.pair) return launch_one<EPI_STORE, 4, true, true>(plan.split, ops, p, st);
    return launch_one<EPI_STORE, 4, true, false>(plan.split, ops, p, st);
  }
  if (plan.pair) return launch_one<EPI_STORE, 4, false, true>(plan.split, ops, p, st);
  if (q_bit == 2) return launch_one<EPI_STORE, 2, false, false>(plan.split, ops, p, st);
  if (q_bit == 8) return launch_one<EPI_STORE, 8, false, false>(plan.split, ops, p, st);
  return launch_one<EPI_STORE, 4, false, false>(plan.split, ops, p, st);
}

// The codes of a CTA's share are decoded at a rate of its own (0.65 us for 64 x 128 elements), so a product on few SMs waits for that, while
// a launch that de-quantizes them uses all.  By the CTAs that the product gets, for 128 rows, us with that launch / decoded inside (cold,
// the launches between a pair of events):
//   K in one CTA: o of 4096 (32 CTAs) 34 / 48; q, k and v of 3072 (72) 38 / 50, of 3328 (78) 42 / 51, of 5120 + 2 x 2560 (80) 61 / 66, of 3584
//     (84) 46 / 54, of 4096 (96) 56 / 59 (one row: 57 / 56), of 5120 (120) 79 / 67; gate and up of 2048 x 5632 (88) 30 / 33, of 2048 x 6400 (100)
//     32 / 33, of 2048 x 8192 (128) 36 / 32, of 4096 x 11008 (172) 92 / 80: five eighths of the SMs.  (K of 8192 and more would pay from 64 on.)
//   K shared by the CTAs of a cluster, and the backward product of down, whose kernel for bf16 weights is the persistent one: down of 2048 x 5632 (64)
//     25.6 / 27.6, of 2560 x 6912 (80) 29.9 / 30.7, of 3072 x 8192 (96) 34.2 / 33.2, of 4096 x 11008 (128) 48 / 40, of 5120 x 13824 (80) 79 / 70; grad_o of
//     2048 (32) 21.5 / 23.6, of 5120 (80) 36 / 37, of 4096 (128) 27.6 / 25.6; grad_x of gate and up of 2048 x 8192 (64) 44 / 46, of 2560 x 6912 (80) 44 / 43;
//     backward of down, 4096 x 8192 (64) 46.0 / 47.5, 4096 x 9728 (76) 49.9 / 48.6, 4096 x 11008 (86) 54 / 48: half of the SMs.
// Without a capture the host has the launch and the allocation to make as well (5 us), and a layer of so few rows waits for the host up to
// widths of 4096 (500 us a step): there only what loses more than that, the products with a fixed order on less than half of the SMs, is
// de-quantized first.  Layer steps of 128 rows, us, by the first lines / by this one: launched 1024 wide 516 to 542 / 485, 2048 520 to 540 / 442 to 500, 3072
// 498 to 523 / 490 to 503; replayed 1024 248 / 274, 2048 331 / 331, 3072 405 / 408.
bool four_pays(int epi, const Params& p, bool recorded) {
  const int split = choose_split(epi, p).split;
  const int ctas = p.N / (epi == EPI_GATEUP ? SBN / 2 : SBN) * (split > 0 ? split : 1);
  if (!recorded) return !p.fixed_order || 2 * ctas >= num_sms();
  return epi == EPI_GRADDOWN || split > 1 ? 2 * ctas >= num_sms() : 8 * ctas >= 5 * num_sms();
}

// the split that a product of up to 128 rows has either way: the same sums for a weight as for its codes
int launch_four(int epi, int q_bit, bool b_mn, const Operands& ops, const Params& p, const FourWeights& four, cudaStream_t st) {
  if (p.M > BM) return HYC_ERR_UNSUPPORTED;
  const SplitPlan plan = choose_split(epi, p);
  const int split = plan.split > 0 ? plan.split : 1;
  if (epi == EPI_GRADDOWN) {
    if (q_bit == 2) return launch_one<EPI_GRADDOWN, 2, true, false, true>(split, ops, p, st, four);
    if (q_bit == 8) return launch_one<EPI_GRADDOWN, 8, true, false, true>(split, ops, p, st, four);
    return launch_one<EPI_GRADDOWN, 4, true, false, true>(split, ops, p, st, four);
  }
  if (epi == EPI_GATEUP) {
    if (q_bit == 2) return launch_one<EPI_GATEUP, 2, false, false, true>(split, ops, p, st, four);
    if (q_bit == 8) return launch_one<EPI_GATEUP, 8, false, false, true>(split, ops, p, st, four);
    return launch_one<EPI_GATEUP, 4, false, false, true>(split, ops, p, st, four);
  }
  if (b_mn) return launch_one<EPI_STORE, 4, true, false, true>(split, ops, p, st, four);
  if (q_bit == 2) return launch_one<EPI_STORE, 2, false, false, true>(split, ops, p, st, four);
  if (q_bit == 8) return launch_one<EPI_STORE, 8, false, false, true>(split, ops, p, st, four);
  return launch_one<EPI_STORE, 4, false, false, true>(split, ops, p, st, four);
}

// Where the line lies (B200, Llama-2-7B weights, us per product, persistent / split):
//   up to 128 tokens, S = the largest of 4, 2, 1 with at most one CTA per SM: x[4096,11008] 42 / 26.5, grad_o 21.8 / 16.6,
//     the three-segment grad_x 67 / 37; unsplit (S = 1) gate/up 48.9 / 43.8, q/k/v 38 / 33.  The grad_down product (bf16
//     weight; as codes it is decoded here) stays persistent: 28.8 / 30.3
//   129 to 256 tokens, pair form, S = 2: 21.8 / 19.0, 43 / 30.6, 69 / 45; wider products fill the chip without it
//   512 tokens: 45 / 47, 75 / 77: persistent
//   (cold L2, each call with its own pair of events, which adds about 5 us: x[4096,11008] of 128 tokens 57 / 35, of 200 tokens
//   51 / 41, grad_o 27 / 23 and 27 / 25)
// A CTA keeps at least 16 k-blocks: below that its share of the main loop is shorter than set-up and reduction (about
// 3 us), and the sum over all of K stays in one accumulator.
// Products whose results the layer quantizes, or that feed tensors it quantizes in the same pass, are not split (gate/up, q/k/v,
// and what the caller marks as such: the o projection): the saved codes of a layer then do not depend through them on how many
// rows are computed together (with 2-bit codes one that flips moves a value by a third of its range).  That leaves 5 us on
// the o projection.  The down projection may be split, so the input of the next layer does depend on it in its last bits.
SplitPlan choose_split(int epi, const Params& p) {
  SplitPlan plan = {0, false};
  if (epi == EPI_GRADDOWN || p.M > 2 * BM) return plan;
  if (epi == EPI_STORE && p.l1.bt != nullptr) return plan;         // a second LoRA term: the persistent kernel's own epilogue
  const int tiles = p.N / (epi == EPI_GATEUP ? SBN / 2 : SBN), sms = num_sms();
  const int kb = (p.K1 + p.K2 + p.K3 + p.K4) / BK;
  const bool whole = epi == EPI_GATEUP || p.q1 != nullptr || p.fixed_order;
  if (whole) {
    if (p.M <= BM && tiles >= sms / 4) plan.split = 1;      // fewer tiles: half-width tiles of the persistent kernel
  } else if (p.M <= BM) {
    plan.split = 1;
    for (int s = 2; s <= 4; s *= 2)
      if (tiles * s <= sms && kb >= 16 * s) plan.split = s;
  } else if (tiles * 4 <= sms && kb >= 32) {
    plan = {2, true};
  }
  return plan;
}

}  // namespace tc
}  // namespace hyc
