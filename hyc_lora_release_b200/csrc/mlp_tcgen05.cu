// tcgen05 / TMEM GEMMs of the LoRA MLP with the activation-compression work in the epilogue.
//
// One persistent kernel, three epilogues:
//   STORE    : D = A * B (+ rank-16 LoRA terms, + residual), bf16 out.  Down projection, grad_x.
//   GATEUP   : [gate_main | up_main] tile = x * [Wg ; Wu]^T, then per element: quantize-and-pack
//              both main branches, add the LoRA terms, SiLU, Hadamard product (forward).
//   GRADDOWN : grad_down tile = g * Wd (+ LoRA), then per element: unpack-dequantize the saved
//              gate/up codes, recompute the forward, emit hadamard, grad_gate, grad_up (backward).
//
// Two CTAs on neighbouring SMs (a cluster of 2) work on one 256 x 256 tile with the pair form of the MMA
// (cta_group::2): CTA r of the pair holds rows 128 r .. 128 r + 127 of the A tile and columns 128 r .. of the
// B tile in its shared memory, the tensor core of each SM reads both halves of B, and each CTA's tensor memory
// receives its own 128 rows of the result.  Per 64-wide k-block an SM therefore pulls 32 KB from L2 instead of
// the 48 KB a 128 x 256 tile of its own would need: the L2-to-SM feed is what bounds the main loop.
//
// Structure of a CTA (320 threads, one CTA per SM, pair tiles dealt round-robin over the pairs):
//   warp 0      : TMA producer (both CTAs): its 128x64 A block and its 128x64 B block per stage (128-byte
//                 swizzle), 6 stages of 32 KB.  The loads of both CTAs complete on the LEADER's (CTA 0 of the
//                 pair) "full" barrier; each CTA waits on its own "empty" barrier.
//   warp 1      : allocates all 512 TMEM columns (two 128x256 fp32 accumulators per CTA; both CTAs take part);
//                 in the leader one lane issues tcgen05.mma.cta_group::2 (M256 N256 K16, bf16 -> fp32) and
//                 commits to the "empty" / "accumulator full" barriers of BOTH CTAs (tcgen05.commit with a CTA
//                 mask; the loads themselves are plain, no multicast).
//   warps 2..9  : epilogue (both CTAs).  Warp w reads TMEM lanes 32*(w%4).. (tcgen05.ld 32x32b.x32) for half
//                 of the tile's columns, so the epilogue of tile i overlaps the MMAs of tile i+1; when a warp
//                 is done with an accumulator it arrives on the leader's "accumulator empty" barrier.
// LoRA terms of the pair form: the epilogue warps first take the whole main branch of the tile into registers and report it
// ("main read"); the MMA warp, between two k-blocks of the next tile, writes the K = 16 products xa B^T into the freed
// columns ("LoRA full"), and the warps come back for them.  grad_down has two terms per column and does this in two rounds.
// The B operand is either K-major ([N,K] row-major, the forward weights) or MN-major ([K,N]
// row-major: the same weights read for the backward products, no transposed copy).
// Every wait is bounded: when a limit is hit the kernel records a code in *status and drains; both CTAs of a
// pair then still meet at the cluster barrier before the tensor memory is released.
// The same kernel also exists without the pairing (template argument PAIR = false: a 128 x 256 tile per CTA,
// 4 stages of 48 KB, cta_group::1 everywhere, no cluster); see launch() for when.
#include "tc_split.cuh"

#ifdef HYC_TC_PROF
#define TC_STAMP(role, it, j) do { if (p.prof != nullptr && blockIdx.x < 2 && (it) < 16) p.prof[blockIdx.x * 384 + ((role) * 16 + (it)) * 8 + (j)] = clock64(); } while (0)
static long long* g_tc_prof = nullptr;
extern "C" __attribute__((visibility("default"))) void hyc_tc_debug_profile(void* buf) { g_tc_prof = (long long*)buf; }
#else
#define TC_STAMP(role, it, j) do { } while (0)
#endif

namespace hyc {
namespace tc {

// first output column of column tile ct
__device__ __forceinline__ int column_tile(int n_wide, int tile_n, int ct) {
  return ct < n_wide ? ct * tile_n : n_wide * tile_n + (ct - n_wide) * (tile_n / 2);
}

// ------------------------------------------------------------------ the kernel
template <int EPI, int QBIT, bool B_MN, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1)
mlp_gemm_kernel(const __grid_constant__ Maps maps, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  uint8_t* stage_base = smem;
  const int stages = p.stages, stage_bytes = p.stage_bytes;
  constexpr int TILE_M = Geo<PAIR>::TILE_M;
  constexpr int B_COLS = Geo<PAIR>::B_COLS;
  __nv_bfloat16* epi_b = reinterpret_cast<__nv_bfloat16*>(smem + PIPE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + PIPE_BYTES + EPI_SMEM_BYTES);
  uint64_t* full = bars;                           // [STAGES]
  uint64_t* empty = bars + MAX_STAGES;             // [STAGES]
  uint64_t* tmem_full = bars + 2 * MAX_STAGES;     // [2]
  uint64_t* tmem_empty = bars + 2 * MAX_STAGES + 2;  // [2]
  uint64_t* main_read = bars + 2 * MAX_STAGES + 4;   // [2] pair form: the main branch of the tile (GRADDOWN: also the first half of
                                                     // the LoRA terms) is in registers, its columns may be overwritten
  uint64_t* lora_full = bars + 2 * MAX_STAGES + 6;   // [2] pair form: LoRA terms are in those columns
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // rank 0: leader of the pair (issues the MMAs), 1: its peer; a CTA on its own is its own leader
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const int pair = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, num_pairs = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int tiles_m = (p.M + TILE_M - 1) / TILE_M;
  constexpr int TILE_N = (EPI == EPI_GATEUP) ? BN / 2 : BN;     // output columns per tile
  const int num_tiles = tiles_m * (p.n_wide + (p.N / TILE_N - p.n_wide) * 2);
  const int kb1 = p.K1 / BK, kb2 = (p.K1 + p.K2) / BK, kb3 = (p.K1 + p.K2 + p.K3) / BK, kb_total = kb3 + p.K4 / BK;

  // pair form: rounds of LoRA products per tile (GRADDOWN has two terms per column and room for one: two rounds)
  const int lora_rounds = !PAIR ? 0 : (EPI == EPI_GATEUP ? 1 : (EPI == EPI_GRADDOWN ? (p.lpre1 == nullptr ? 2 : 0) : (p.l0.bt != nullptr ? 1 : 0)));
  LoraStage lst;
  lst.a1 = smem + PIPE_BYTES + 16384; lst.a2 = lst.a1 + 4096; lst.b1 = lst.a1 + 8192; lst.b2 = lst.a1 + 12288;

  if (warp == 0 && elect_one()) {
    for (int i = 0; i < 3; ++i) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.a[i])) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.b[i])) : "memory");
    }
  }
  if (threadIdx.x == 0) {
    // full / tmem_empty are used in the leader only: the loads of both CTAs and the epilogue warps of both CTAs
    // arrive there; empty / tmem_full exist in both CTAs and are signalled together by the leader's commits
    for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], (PAIR ? 2 : 1) * EPI_WARPS);
      mbar_init(&main_read[b], 2 * EPI_WARPS); mbar_init(&lora_full[b], 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();      // before tensor memory is taken: see launch_pdl
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the peer's barriers are initialised before anything is signalled there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int pit = 0;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++pit) {
        const int m0 = (tile % tiles_m) * TILE_M + (int)rank * BM, ct = tile / tiles_m;
        const bool wide = ct < p.n_wide;
        const int nt = column_tile(p.n_wide, TILE_N, ct), b_cols = wide ? B_COLS : B_COLS / 2;
        const int grp = nt < p.g_end0 ? 0 : (nt < p.g_end1 ? 1 : 2);
        const int n0 = nt - (grp == 0 ? 0 : (grp == 1 ? p.g_end0 : p.g_end1));
        TC_STAMP(0, pit, 0);
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait_warp(&empty[stage], phase ^ 1u, abort_flag)) {
            if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_PRODUCER); }
            ok = false;
            break;
          }
          const int seg = kb < kb1 ? 0 : (kb < kb2 ? 1 : (kb < kb3 ? 2 : 3));
          const int wsel = EPI == EPI_STORE && grp > 0 ? grp : seg;      // weights side by side along N, or K segments
          const CUtensorMap* ma = &maps.a[seg];
          const CUtensorMap* mb = wide ? &maps.b[wsel] : &maps.n[wsel];
          const int k0 = (kb - (seg == 0 ? 0 : (seg == 1 ? kb1 : (seg == 2 ? kb2 : kb3)))) * BK;
          const uint32_t sa = smem_u32(stage_base + stage * stage_bytes);
          const uint32_t sb = sa + STAGE_A_BYTES;
          // pair form: the leader's barrier counts both CTAs' bytes
          const uint32_t fbar = PAIR ? map_to_cta(&full[stage], 0) : smem_u32(&full[stage]);
          if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&full[stage], (uint32_t)((PAIR ? 2 : 1) * (STAGE_A_BYTES + b_cols * BK * 2)));
          tma_load_2d<PAIR>(sa, ma, fbar, k0, m0);
          // B: K-major in one box of 128 weight rows (64 for a narrow tile), MN-major in boxes of 64 x 64.  Unrolled and
          // predicated: a loop with a run-time count here cost the K-long products 10 %, two 64-row boxes instead of
          // one of 128 rows 5 %
          const int box = wide ? 128 : 64;
          if (EPI == EPI_GATEUP) {
            // the first half of the tile's B columns are rows of Wg, the second half the same rows of Wu (pair form: the
            // leader fetches the former, the peer the latter)
            const CUtensorMap* mg = wide ? &maps.b[0] : &maps.n[0];
            const CUtensorMap* mu = wide ? &maps.b[1] : &maps.n[1];
            if (PAIR) {
              tma_load_2d<PAIR>(sb, rank == 0 ? mg : mu, fbar, k0, n0);
            } else {
              tma_load_2d<PAIR>(sb, mg, fbar, k0, n0);
              tma_load_2d<PAIR>(sb + box * 128, mu, fbar, k0, n0);
            }
          } else if (B_MN) {
            const int nb = n0 + (int)rank * b_cols;
#pragma unroll
            for (int j = 0; j < B_COLS / 64; ++j)
              if (j < B_COLS / 128 || wide) tma_load_2d<PAIR>(sb + j * 8192, mb, fbar, nb + 64 * j, k0);
          } else {
            tma_load_2d<PAIR>(sb, mb, fbar, k0, n0 + (int)rank * b_cols);
            if (!PAIR) tma_load_2d<PAIR>(sb + box * 128, mb, fbar, k0, n0 + box);
          }
          }
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        TC_STAMP(0, pit, 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0) {
      // instruction descriptor: fp32 accumulate, bf16 x bf16, M = 256 (the pair) or 128, N = 256 or 128, B major as given
      const uint32_t idesc_any = (1u << 4) | (1u << 7) | (1u << 10) | ((B_MN ? 1u : 0u) << 16) | ((uint32_t)(TILE_M >> 4) << 24);
      const uint32_t idesc_wide = idesc_any | ((uint32_t)(BN >> 3) << 17), idesc_narrow = idesc_any | ((uint32_t)(BN >> 4) << 17);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      // LoRA products of the tile before: due as soon as the epilogue has taken its main branch out, so between the k-blocks
      // of the present tile
      int due = 0, due_buf = 0, due_cols = 0;
      uint32_t due_parity = 0u;             // one bit per accumulator
      auto lora_products = [&](bool wait) {
        while (due > 0) {
          if (wait) {
            if (!mbar_wait_warp(&main_read[due_buf], (due_parity >> due_buf) & 1u, abort_flag)) {
              if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_MMA); }
              return false;
            }
          } else if (!__all_sync(0xffffffffu, mbar_test(&main_read[due_buf], (due_parity >> due_buf) & 1u))) {
            return true;
          }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t d = tmem_base + (uint32_t)(due_buf * BN);
            // columns of one product; GRADDOWN takes a quarter of the tile's columns from each CTA's operand per round
            const int n = EPI == EPI_GRADDOWN ? due_cols / 2 : due_cols;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TILE_M >> 4) << 24) | ((uint32_t)(n >> 3) << 17);
            const uint32_t b_off = EPI == EPI_GRADDOWN && due == 1 ? k16_offset(due_cols / 4, 0) : 0u;
            tc_mma<PAIR>(d, make_desc_k16(smem_u32(lst.a1)), make_desc_k16(smem_u32(lst.b1) + b_off), idesc, 0u);
            if (EPI != EPI_STORE) tc_mma<PAIR>(d + (uint32_t)n, make_desc_k16(smem_u32(lst.a2)), make_desc_k16(smem_u32(lst.b2) + b_off), idesc, 0u);
            tc_commit<PAIR>(&lora_full[due_buf]);
          }
          __syncwarp();
          due_parity ^= 1u << due_buf;
          --due;
        }
        return true;
      };
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++it) {
        const uint32_t idesc = tile / tiles_m < p.n_wide ? idesc_wide : idesc_narrow;
        const int buf = it & 1;
        const uint32_t bphase = (uint32_t)(it >> 1) & 1u;
        TC_STAMP(1, it, 0);
        if (!mbar_wait_warp(&tmem_empty[buf], bphase ^ 1u, abort_flag)) {
          if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_MMA); }
          break;
        }
        tc_fence_after();
        TC_STAMP(1, it, 1);
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait_warp(&full[stage], phase, abort_flag)) {
            if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_MMA); }
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(stage_base + stage * stage_bytes);
          const uint32_t sb = sa + STAGE_A_BYTES;
          const uint64_t adesc = make_desc(sa, 16, 1024);
          const uint64_t bdesc = B_MN ? make_desc(sb, 64 * 128, 1024) : make_desc(sb, 16, 1024);
          if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            // K-major: 16 elements = 32 bytes further along the swizzled row; MN-major: 16 k-rows of 128 bytes
            const uint64_t a = adesc + (uint64_t)(kk * 2);
            const uint64_t b = bdesc + (uint64_t)(B_MN ? kk * 128 : kk * 2);
            tc_mma<PAIR>(d_tmem, a, b, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          }
          tc_commit<PAIR>(&empty[stage]);
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1u; }
          if (PAIR && due > 0) lora_products(false);
        }
        if (ok && elect_one()) tc_commit<PAIR>(&tmem_full[buf]);
        __syncwarp();
        if (PAIR) {
          // what is left of the tile before: its accumulator is the next one to be written
          if (ok && !lora_products(true)) ok = false;
          due = lora_rounds; due_buf = buf; due_cols = tile / tiles_m < p.n_wide ? TILE_N : TILE_N / 2;
        }
        TC_STAMP(1, it, 2);
      }
      if (PAIR && ok) lora_products(true);
    }
  } else {
    // ------------------------------------------------ epilogue warps
    const int et = threadIdx.x - 64;
    const int quad = warp & 3;
    const int chalf = (warp - 2) >> 2;
    // scratch of the epilogue warps (layout: see EPI_SMEM_BYTES)
    uint32_t* sR1 = reinterpret_cast<uint32_t*>(epi_b) + (warp - 2) * 1024;      // this warp's two tiles
    uint32_t* sR2 = sR1 + 512;
    float* sGV = reinterpret_cast<float*>(epi_b) + 2 * BN * 16;   // STORE: BN quantizer constants; GATEUP: two vectors of BN/2
    __nv_bfloat16* sGS = reinterpret_cast<__nv_bfloat16*>(sGV);   // GRADDOWN: two bf16 scale vectors of BN
    int it = 0;
    const uint32_t tmem_empty_leader[2] = {PAIR ? map_to_cta(&tmem_empty[0], 0) : smem_u32(&tmem_empty[0]),
                                           PAIR ? map_to_cta(&tmem_empty[1], 0) : smem_u32(&tmem_empty[1])};
    bool fine = true;                    // false: a wait gave up; the barriers below are still kept
    if constexpr (PAIR) {
      uint32_t* R = reinterpret_cast<uint32_t*>(epi_b) + (warp - 2) * 512;      // this warp's tile
      const uint32_t main_read_leader = map_to_cta(&main_read[0], 0);
      uint32_t lora_parity = 0u;           // one bit per accumulator
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (fine && !mbar_wait(bar, parity, abort_flag)) {
          if (!*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_EPILOGUE); }
          fine = false;
        }
        fine = __all_sync(0xffffffffu, fine);
        tc_fence_after();
      };
      for (int tile = pair; tile < num_tiles; tile += num_pairs, ++it) {
        const int m0 = (tile % tiles_m) * TILE_M + (int)rank * BM, ct = tile / tiles_m;
        const bool wide = ct < p.n_wide;
        const int n0 = column_tile(p.n_wide, TILE_N, ct), cols = wide ? TILE_N : TILE_N / 2;
        const int buf = it & 1;
        const int64_t row0 = (int64_t)m0 + quad * 32, row = row0 + lane;
        const bool valid = row < p.M;
        const int cb0 = cols / 2 * chalf, blocks = cols / 64;                   // this warp's columns of the tile, in blocks of 32
        const StoreView sv = store_view(p, n0);
        // ---- constants and LoRA operands of the tile (the readers of the previous ones are done: barrier at the end)
        if (EPI == EPI_STORE) {
          if (sv.q != nullptr && et < cols) sGV[et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(sv.s[sv.n0 + et])));
          if (lora_rounds) {
            stage_lora_a(lst.a1, sv.l0.xa, m0, p.M, et);
            stage_lora_b(lst.b1, sv.l0, sv.n0 + (int)rank * (cols / 2), cols / 2, et);
          }
        } else if (EPI == EPI_GATEUP) {
          if (et < cols) {
            sGV[et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(p.s1[n0 + et])));
            sGV[BN / 2 + et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(p.s2[n0 + et])));
          }
        } else if (et < cols) {      // the scales stay bf16: column pairs are read as one packed word
          sGS[et] = p.s1[n0 + et];
          sGS[BN + et] = p.s2[n0 + et];
        }
        if (EPI != EPI_STORE && lora_rounds) {
          const LoraTerm &la = EPI == EPI_GATEUP ? p.l0 : p.l1, &lb = EPI == EPI_GATEUP ? p.l1 : p.l2;
          stage_lora_a(lst.a1, la.xa, m0, p.M, et);
          stage_lora_a(lst.a2, lb.xa, m0, p.M, et);
          stage_lora_b(lst.b1, la, n0 + (int)rank * (cols / 2), cols / 2, et);
          stage_lora_b(lst.b2, lb, n0 + (int)rank * (cols / 2), cols / 2, et);
        }
        if (lora_rounds) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        uint4 res[4];                        // STORE: the residual of the next block
        GdCodes<QBIT> codes;                 // GRADDOWN: codes of the next block
        if (EPI == EPI_STORE && sv.residual != nullptr) tile_fetch(sv.residual, row0, p.M, sv.ld, (int64_t)sv.n0 + cb0, lane, res);
        if (EPI == EPI_GRADDOWN) gd_codes<QBIT>(p, row, (int64_t)n0 + cb0, codes);
        epi_bar_sync();
        wait(&tmem_full[buf], (uint32_t)(it >> 1) & 1u);
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN);
        auto columns_read = [&]() {          // what this warp needed of the accumulator is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(main_read_leader + 8u * (uint32_t)buf);
        };
        auto lora_wait = [&]() {
          wait(&lora_full[buf], (lora_parity >> buf) & 1u);
          lora_parity ^= 1u << buf;
        };
        if (fine) {
          if constexpr (EPI == EPI_GATEUP) {
            uint32_t xg[2][16], xu[2][16];
#pragma unroll
            for (int b = 0; b < 2; ++b)
              if (b < blocks) {
                tc_ld_pairs(t_lane + (uint32_t)(cb0 + 32 * b), xg[b]);
                tc_ld_pairs(t_lane + (uint32_t)(cols + cb0 + 32 * b), xu[b]);
              }
            columns_read();
            // the codes while the LoRA products wait their turn on the tensor pipe
#pragma unroll
            for (int b = 0; b < 2; ++b)
              if (b < blocks) {
                const int64_t n = (int64_t)n0 + cb0 + 32 * b;
                uint32_t w1[BlockGeo<QBIT>::NW], w2[BlockGeo<QBIT>::NW];
                pack_codes<QBIT>(xg[b], sGV + cb0 + 32 * b, w1);
                pack_codes<QBIT>(xu[b], sGV + BN / 2 + cb0 + 32 * b, w2);
                if (valid) {
                  store_block_words<QBIT>(p.q1 + (row * p.N + n) * QBIT / 8, w1);
                  store_block_words<QBIT>(p.q2 + (row * p.N + n) * QBIT / 8, w2);
                  if (p.dbg1 != nullptr) { store_pairs(xg[b], p.dbg1 + row * p.N + n); store_pairs(xu[b], p.dbg2 + row * p.N + n); }
                }
              }
            lora_wait();
#pragma unroll
            for (int b = 0; b < 2; ++b)
              if (b < blocks) {
                uint32_t l1[16], l2[16];
                tc_ld_pairs(t_lane + (uint32_t)(cb0 + 32 * b), l1);
                tc_ld_pairs(t_lane + (uint32_t)(cols + cb0 + 32 * b), l2);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const uint32_t y1 = add2(xg[b][i], l1[i]);
                  l1[i] = mul2(mul2(y1, sigmoid2(y1)), add2(xu[b][i], l2[i]));
                }
                flush_pairs(l1, R, p.out0, row0, p.M, p.N, (int64_t)n0 + cb0 + 32 * b, lane);
              }
          } else if constexpr (EPI == EPI_GRADDOWN) {
            uint32_t gd[4][16];
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < blocks) tc_ld_pairs(t_lane + (uint32_t)(cb0 + 32 * b), gd[b]);
            if (lora_rounds) columns_read();
            // round r: blocks r * blocks / 2 ..; the first half of the tile's columns hold the gate terms of both column halves, the
            // second half the up terms
            const int per = blocks / 2;
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < blocks) {
                const int64_t n = (int64_t)n0 + cb0 + 32 * b;
                const GdCodes<QBIT> cur = codes;
                if (b + 1 < blocks) gd_codes<QBIT>(p, row, n + 32, codes);
                uint32_t t1[16], t2[16], o[16];
                if (lora_rounds) {
                  if (b == 0 || b == per) lora_wait();
                  const uint32_t at = t_lane + (uint32_t)(chalf * (cols / 4) + 32 * (b < per ? b : b - per));
                  tc_ld_pairs(at, t1);
                  tc_ld_pairs(at + (uint32_t)(cols / 2), t2);
                  if (b == per - 1) columns_read();
                } else {
#pragma unroll
                  for (int c8 = 0; c8 < 4; ++c8) {      // the terms of a launch that prepared them
                    uint4 a = make_uint4(0u, 0u, 0u, 0u), c = a;
                    if (valid) {
                      a = *reinterpret_cast<const uint4*>(p.lpre1 + row * p.ld_pre + n + 8 * c8);
                      c = *reinterpret_cast<const uint4*>(p.lpre2 + row * p.ld_pre + n + 8 * c8);
                    }
                    t1[4 * c8] = a.x; t1[4 * c8 + 1] = a.y; t1[4 * c8 + 2] = a.z; t1[4 * c8 + 3] = a.w;
                    t2[4 * c8] = c.x; t2[4 * c8 + 1] = c.y; t2[4 * c8 + 2] = c.z; t2[4 * c8 + 3] = c.w;
                  }
                }
                const uint32_t* sS1 = reinterpret_cast<const uint32_t*>(sGS) + (cb0 + 32 * b) / 2;
                const uint32_t* sS2 = reinterpret_cast<const uint32_t*>(sGS + BN) + (cb0 + 32 * b) / 2;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const uint32_t x1 = dequant_pair<QBIT>(cur.w1, 2 * i, sS1[i]), x2 = dequant_pair<QBIT>(cur.w2, 2 * i, sS2[i]);
                  const uint32_t y1 = add2(x1, t1[i]), sig = sigmoid2(y1), y1s = mul2(y1, sig), y2 = add2(x2, t2[i]);
                  o[i] = mul2(y1s, y2);
                  const uint32_t inner = add2(kOne2, mul2(y1, sub2(kOne2, sig)));
                  t1[i] = mul2(mul2(gd[b][i], y2), mul2(sig, inner));
                  t2[i] = mul2(gd[b][i], y1s);
                }
                flush_pairs(o, R, p.out0, row0, p.M, p.N, n, lane);
                flush_pairs(t1, R, p.out1, row0, p.M, p.N, n, lane);
                flush_pairs(t2, R, p.out2, row0, p.M, p.N, n, lane);
              }
          } else {
            const bool has1 = sv.l1.bt != nullptr, has_res = sv.residual != nullptr;
            uint32_t x[4][16];
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < blocks) tc_ld_pairs(t_lane + (uint32_t)(cb0 + 32 * b), x[b]);
            if (lora_rounds) columns_read();
            if (sv.q != nullptr || sv.main != nullptr) {
#pragma unroll
              for (int b = 0; b < 4; ++b)
                if (b < blocks && valid) {
                  const int64_t n = (int64_t)sv.n0 + cb0 + 32 * b;
                  if (sv.q != nullptr) {
                    uint32_t w1[BlockGeo<QBIT>::NW];
                    pack_codes<QBIT>(x[b], sGV + cb0 + 32 * b, w1);
                    store_block_words<QBIT>(sv.q + (row * sv.ld + n) * QBIT / 8, w1);
                  }
                  if (sv.main != nullptr) store_pairs(x[b], sv.main + row * sv.ld + n);
                }
            }
            if (lora_rounds) lora_wait();
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < blocks) {
                const int64_t n = (int64_t)sv.n0 + cb0 + 32 * b;
                if (lora_rounds) {
                  uint32_t l[16];
                  tc_ld_pairs(t_lane + (uint32_t)(cb0 + 32 * b), l);
#pragma unroll
                  for (int i = 0; i < 16; ++i) x[b][i] = add2(x[b][i], l[i]);
                }
                if (has1) {
#pragma unroll 1
                  for (int i = 0; i < 16; ++i) {
                    const uint32_t l = pack_bf16x2_rn(lora_dot_global(sv.l1, n + 2 * i, row, valid), lora_dot_global(sv.l1, n + 2 * i + 1, row, valid));
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                      if (j == i) x[b][j] = add2(x[b][j], l);
                  }
                }
                if (has_res) {
                  const uint4 now[4] = {res[0], res[1], res[2], res[3]};
                  if (b + 1 < blocks) tile_fetch(sv.residual, row0, p.M, sv.ld, n + 32, lane, res);
                  tile_put(R, lane, now);
                  __syncwarp();
#pragma unroll
                  for (int c8 = 0; c8 < 4; ++c8) {
                    const uint4 r = *reinterpret_cast<const uint4*>(R + gd_chunk(lane, c8));
                    x[b][4 * c8] = add2(x[b][4 * c8], r.x); x[b][4 * c8 + 1] = add2(x[b][4 * c8 + 1], r.y);
                    x[b][4 * c8 + 2] = add2(x[b][4 * c8 + 2], r.z); x[b][4 * c8 + 3] = add2(x[b][4 * c8 + 3], r.w);
                  }
                  __syncwarp();
                }
                flush_pairs(x[b], R, sv.out, row0, p.M, sv.ld, n, lane);
              }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(tmem_empty_leader[buf]);
        epi_bar_sync();    // everyone is done with the staged tile before the next one overwrites it
      }
    } else
    for (int tile = pair; tile < num_tiles; tile += num_pairs, ++it) {
      const int m0 = (tile % tiles_m) * TILE_M + (int)rank * BM, ct = tile / tiles_m;
      const bool wide = ct < p.n_wide;
      const int n0 = column_tile(p.n_wide, TILE_N, ct), cols = wide ? TILE_N : TILE_N / 2;
      const int buf = it & 1;
      const uint32_t bphase = (uint32_t)(it >> 1) & 1u;
      const int64_t row0 = (int64_t)m0 + quad * 32;
      if (et == 0) TC_STAMP(2, it, 0);

      // stage the per-tile constants (previous tile's readers are done: barrier at the end)
      const StoreView sv = store_view(p, n0);
      const int cb0 = cols / 2 * chalf, cb_end = cols / 2 * (chalf + 1);      // this warp's columns of the tile
      LoraA a1, a2;                        // the warp's LoRA-A rows
      LoraB b1, b2;                        // LoRA-B columns of the next block, fetched one block ahead
      uint4 res[4];                        // STORE: the residual of the next block
      GdInputs<QBIT> gin;                  // GRADDOWN: codes and LoRA-B columns of the next block
      if (EPI == EPI_STORE) {
        if (sv.q != nullptr && et < cols) sGV[et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(sv.s[sv.n0 + et])));
        if (sv.l0.bt != nullptr) {
          lora_load_a(sv.l0.xa, row0, p.M, lane, a1);
          lora_load_b(sv.l0, (int64_t)sv.n0 + cb0, lane, b1);
        }
        if (sv.residual != nullptr) tile_fetch(sv.residual, row0, p.M, sv.ld, (int64_t)sv.n0 + cb0, lane, res);
      } else if (EPI == EPI_GATEUP) {
        if (et < cols) {
          sGV[et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(p.s1[n0 + et])));
          sGV[BN / 2 + et] = fastq_scale<QBIT>(__frcp_rn(__bfloat162float(p.s2[n0 + et])));
        }
        lora_load_a(p.l0.xa, row0, p.M, lane, a1);
        lora_load_a(p.l1.xa, row0, p.M, lane, a2);
        lora_load_b(p.l0, (int64_t)n0 + cb0, lane, b1);
        lora_load_b(p.l1, (int64_t)n0 + cb0, lane, b2);
      } else {
        // the scales stay bf16: column pairs are read as one packed word
        if (et < cols) {
          sGS[et] = p.s1[n0 + et];
          sGS[BN + et] = p.s2[n0 + et];
        }
        lora_load_a(p.l1.xa, row0, p.M, lane, a1);
        lora_load_a(p.l2.xa, row0, p.M, lane, a2);
        // the first block's inputs are on their way while the warp waits for the accumulator
        gd_fetch<QBIT>(p, row0, lane, (int64_t)n0 + cb0, gin);
      }
      epi_bar_sync();
      if (et == 0) TC_STAMP(2, it, 1);

      if (fine && !mbar_wait(&tmem_full[buf], bphase, abort_flag)) {
        if (!*abort_flag) { *abort_flag = 1; atomicExch(p.status, ST_TIMEOUT_EPILOGUE); }
        fine = false;
      }
      fine = __all_sync(0xffffffffu, fine);
      tc_fence_after();
      if (et == 0) TC_STAMP(2, it, 2);
      const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN);
      if (fine) {
        // GATEUP: gate columns, then the up columns of the accumulator; a warp takes half of each
#pragma unroll 1
        for (int cb = cb0; cb < cb_end; cb += 32) {
          const bool more = cb + 32 < cb_end;
          uint32_t acc[32];
          tc_ld32(t_lane + (uint32_t)cb, acc);
          if (EPI == EPI_GATEUP) {
            uint32_t u[32];
            tc_ld32(t_lane + (uint32_t)(cols + cb), u);
            const LoraB n1 = b1, n2 = b2;
            if (more) {
              lora_load_b(p.l0, (int64_t)n0 + cb + 32, lane, b1);
              lora_load_b(p.l1, (int64_t)n0 + cb + 32, lane, b2);
            }
            epi_gateup_block<QBIT>(p, row0, lane, n0, cb, acc, u, a1, a2, n1, n2, sGV, sGV + BN / 2, sR1, sR2);
          } else if (EPI == EPI_STORE) {
            const uint4 now[4] = {res[0], res[1], res[2], res[3]};
            const LoraB n1 = b1;
            if (more && sv.residual != nullptr) tile_fetch(sv.residual, row0, p.M, sv.ld, (int64_t)sv.n0 + cb + 32, lane, res);
            if (more && sv.l0.bt != nullptr) lora_load_b(sv.l0, (int64_t)sv.n0 + cb + 32, lane, b1);
            epi_store_block<QBIT>(sv, row0, lane, p.M, cb, acc, a1, n1, sGV, now, sR1, sR2);
          } else {
            const GdInputs<QBIT> cur = gin;
            if (more) gd_fetch<QBIT>(p, row0, lane, (int64_t)n0 + cb + 32, gin);
            epi_graddown_block<QBIT>(p, row0, lane, n0, cb, acc, cur, a1, a2, sR1, sR2,
                                     reinterpret_cast<const uint32_t*>(sGS), reinterpret_cast<const uint32_t*>(sGS + BN));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (et == 0) TC_STAMP(2, it, 3);
      if (lane == 0) mbar_arrive_cluster(tmem_empty_leader[buf]);
      epi_bar_sync();    // everyone is done with the staged tile before the next one overwrites it
      if (et == 0) TC_STAMP(2, it, 4);
    }
  }

  // ------------------------------------------------ teardown
  // both CTAs are done with each other's barriers and tensor memory before either leaves
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// Of `columns` full-width column tiles, how many stay full width so that `units` workers that take the tiles in turn
// (wide ones first) finish earliest.  A half-width tile costs 0.68 of a full one: the A block is loaded all the same (one round
// of half-width against one of full-width tiles on 74 pairs, 256 and 512 rows, K 4096 and 11008, both forms of B: 0.64 to
// 0.72, mean 0.69).
static int choose_wide(int tiles_m, int columns, int units) {
  int best = columns;
  float best_cost = 1e30f;
  const float half = 0.68f;
  for (int w = columns; w >= 0; --w) {
    const int wide = tiles_m * w, narrow = tiles_m * 2 * (columns - w);
    const int rounds = wide / units, rest = wide % units;            // the first `rest` workers have one wide tile more
    const int behind = narrow - (units - rest);                      // narrow tiles left when those come round
    float cost = rounds + half * ((narrow + units - 1) / units);
    if (rest > 0) {
      const float c0 = rounds + 1 + half * (behind > 0 ? (behind + units - 1) / units : 0);
      if (c0 > cost) cost = c0;
    }
    if (cost < best_cost - 0.02f) { best_cost = cost; best = w; }
  }
  return best;
}

template <int EPI, int QBIT, bool B_MN, bool PAIR>
static int launch_as(const Operands& ops, const Params& p, cudaStream_t st) {
  auto kern = mlp_gemm_kernel<EPI, QBIT, B_MN, PAIR>;
  // the attribute belongs to a (function, device) pair: set once per device (unknown device: every time)
  static bool attr[64] = {false};
  const int slot = current_device_slot();
  if (slot < 0 || !attr[slot]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) {
      hyc_set_last_cuda_error((int)cudaGetLastError());
      return HYC_ERR_LAUNCH;
    }
    if (slot >= 0) attr[slot] = true;
  }
  constexpr int TILE_N = (EPI == EPI_GATEUP) ? BN / 2 : BN;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 2; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = PAIR ? 2 : 1;
  // the kernel is persistent: one CTA per SM, or one pair per two neighbouring SMs (as many as can be resident)
  int units = num_sms();
  if (PAIR) {
    static int pairs_on[64] = {0};
    int pairs = slot >= 0 ? pairs_on[slot] : 0;
    if (pairs == 0) {
      cfg.gridDim = dim3(2 * (unsigned)(num_sms() / 2));
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = num_sms() / 2; }
      pairs = n < num_sms() / 2 ? n : num_sms() / 2;
      if (pairs < 1) pairs = 1;
      if (slot >= 0) pairs_on[slot] = pairs;
    }
    units = pairs;
  }
  Params pp = p;
  const int tiles_m = (p.M + Geo<PAIR>::TILE_M - 1) / Geo<PAIR>::TILE_M, columns = p.N / TILE_N;
  pp.n_wide = choose_wide(tiles_m, columns, units);
  // half-width tiles only: the B part of a stage is half as big and the ring has more stages
  pp.stage_bytes = STAGE_A_BYTES + Geo<PAIR>::STAGE_B_BYTES / (pp.n_wide == 0 ? 2 : 1);
  pp.stages = PIPE_BYTES / pp.stage_bytes < MAX_STAGES ? PIPE_BYTES / pp.stage_bytes : MAX_STAGES;
  const int tiles = tiles_m * (pp.n_wide + 2 * (columns - pp.n_wide));
  cfg.gridDim = dim3((unsigned)((PAIR ? 2 : 1) * (tiles < units ? tiles : units)));
#ifdef HYC_TC_PROF
  pp.prof = g_tc_prof;
#endif
  Maps maps;
  if (!make_maps(&maps, ops, B_MN, BM, 128, pp.n_wide < columns)) return HYC_ERR_UNSUPPORTED;
  if (cudaLaunchKernelEx(&cfg, kern, maps, pp) != cudaSuccess) {
    hyc_set_last_cuda_error((int)cudaGetLastError());
    return HYC_ERR_LAUNCH;
  }
  return HYC_OK;
}

template <int EPI, int QBIT, bool B_MN>
static int launch(const Operands& ops, const Params& p, cudaStream_t st, const FourWeights* four = nullptr) {
  if (four != nullptr) return launch_four(EPI, QBIT, B_MN, ops, p, *four, st);
  const SplitPlan plan = choose_split(EPI, p);
  if (plan.split > 0) return launch_split(EPI, QBIT, B_MN, plan, ops, p, st);
  // pairs, except where few rows would leave half of the tile empty
  bool pair = p.M > BM;
  return pair ? launch_as<EPI, QBIT, B_MN, true>(ops, p, st) : launch_as<EPI, QBIT, B_MN, false>(ops, p, st);
}

}  // namespace tc
}  // namespace hyc

using namespace hyc;
using namespace hyc::tc;

static constexpr int kGemmForms = HYC_GEMM_B_KN | HYC_GEMM_FIXED_ORDER;

static LoraTerm make_term(const void* xa, const void* bt, int64_t ld_col, int64_t ld_r) {
  LoraTerm t;
  t.xa = (const __nv_bfloat16*)xa;
  t.bt = (const __nv_bfloat16*)bt;
  t.ld_col = ld_col;
  t.ld_r = ld_r;
  return t;
}

// the weights of a product as the split kernel decodes them; `w`: null, or one entry per B operand (its `packed` null: that one is bf16)
static int shift_of(int blocksize) {
  int s = 0;
  while ((1 << s) < blocksize && s < 30) ++s;
  return (1 << s) == blocksize ? s : -1;
}
static bool four_takes(const hyc_nf4_weight& w, int rows, int cols) {
  if (!w.packed || !w.code16 || (!w.absmax && (!w.absmax_q || !w.code256 || !w.absmax2))) return false;
  return rows >= 1 && rows <= BM && cols % 64 == 0 && w.blocksize >= 64 && shift_of(w.blocksize) >= 0 && aligned(w.packed, 32) && aligned(w.code16, 4) &&
         (w.absmax || (w.blocksize2 >= 1 && shift_of(w.blocksize2) >= 0));
}
static FourView four_view(const hyc_nf4_weight& w, int64_t cols) {
  return {(const uint8_t*)w.packed, w.code16, w.absmax, w.absmax_q, w.code256, w.absmax2, cols, shift_of(w.blocksize),
          w.absmax ? 0 : shift_of(w.blocksize2), w.offset};
}
static bool has_four(const hyc_nf4_weight* w, int i) { return w != nullptr && w[i].packed != nullptr; }
// (a product whose operands are all bf16 is its namesake's, with any number of rows)
static bool any_four(const hyc_nf4_weight* w, int count) {
  for (int i = 0; i < count; ++i)
    if (has_four(w, i)) return true;
  return false;
}

extern "C" HYC_API int hyc_nf4_product_supported(const hyc_nf4_weight* w, int rows, int cols) { return w && four_takes(*w, rows, cols) ? 1 : 0; }
extern "C" HYC_API int hyc_nf4_product_pays(int kind, int rows, int n, int k, int recorded) {
  if (rows < 1 || rows > BM || n < 1 || k < 1) return 0;
  Params p = {};
  p.M = rows; p.N = n; p.K1 = k;
  p.fixed_order = kind == HYC_GEMM_FIXED_ORDER;
  return four_pays(kind == HYC_NF4_GATE_UP ? EPI_GATEUP : (kind == HYC_NF4_GRAD_DOWN ? EPI_GRADDOWN : EPI_STORE), p, recorded != 0) ? 1 : 0;
}

extern "C" HYC_API int hyc_gemm_bf16_tcgen05(
    const void* A, const void* B, int M, int N, int K, int form,
    const void* A2, const void* B2, int K2, const void* A3, const void* B3, int K3,
    const void* xa0, const void* bt0, int64_t bt0_ld_col, int64_t bt0_ld_r,
    const void* xa1, const void* bt1, int64_t bt1_ld_col, int64_t bt1_ld_r,
    const void* residual, void* D, int* status, void* stream) {
  if (!A || !B || !D || !status) return HYC_ERR_NULL;
  if (form & ~kGemmForms) return HYC_ERR_SHAPE;
  const bool b_is_kn = (form & HYC_GEMM_B_KN) != 0;
  if ((K2 > 0) != (A2 != nullptr && B2 != nullptr)) return HYC_ERR_NULL;
  if ((K3 > 0) != (A3 != nullptr && B3 != nullptr)) return HYC_ERR_NULL;
  if (M <= 0 || N <= 0 || K <= 0 || N % BN != 0 || K % BK != 0 || K2 < 0 || K2 % BK != 0 || K3 < 0 || K3 % BK != 0)
    return HYC_ERR_SHAPE;
  if (!aligned(A, 16) || !aligned(B, 16) || !aligned(D, 16) || (residual && !aligned(residual, 16)) ||
      (xa0 && !aligned(xa0, 16)) || (xa1 && !aligned(xa1, 16)) || (A2 && (!aligned(A2, 16) || !aligned(B2, 16))) ||
      (A3 && (!aligned(A3, 16) || !aligned(B3, 16)))) return HYC_ERR_ALIGN;
  if ((bt0 != nullptr) != (xa0 != nullptr) || (bt1 != nullptr) != (xa1 != nullptr)) return HYC_ERR_NULL;
  Operands ops = {};
  ops.a[0] = {A, M, K};
  ops.b[0] = b_is_kn ? Matrix{B, K, N} : Matrix{B, N, K};
  if (K2 > 0) { ops.a[1] = {A2, M, K2}; ops.b[1] = b_is_kn ? Matrix{B2, K2, N} : Matrix{B2, N, K2}; }
  if (K3 > 0) { ops.a[2] = {A3, M, K3}; ops.b[2] = b_is_kn ? Matrix{B3, K3, N} : Matrix{B3, N, K3}; }
  Params p = {};
  p.M = M; p.N = N; p.K1 = K; p.K2 = K2; p.K3 = K3; p.epi = EPI_STORE; p.q_bit = 0;
  p.fixed_order = (form & HYC_GEMM_FIXED_ORDER) != 0;
  p.l0 = make_term(xa0, bt0, bt0_ld_col, bt0_ld_r);
  p.l1 = make_term(xa1, bt1, bt1_ld_col, bt1_ld_r);
  p.l2 = make_term(nullptr, nullptr, 0, 0);
  p.residual = (const __nv_bfloat16*)residual;
  p.out0 = (__nv_bfloat16*)D;
  p.status = status;
  p.g_end0 = p.g_end1 = N;
  cudaStream_t st = (cudaStream_t)stream;
  return b_is_kn ? launch<EPI_STORE, 4, true>(ops, p, st) : launch<EPI_STORE, 4, false>(ops, p, st);
}

static int gemm_segments(int count, const void* const* A, const void* const* B, const hyc_nf4_weight* B4, const int* K, int M, int N,
                         int form, const void* residual, void* D, int* status, void* stream) {
  if (!A || !B || !K || !D || !status) return HYC_ERR_NULL;
  if (form & ~kGemmForms) return HYC_ERR_SHAPE;
  const bool b_is_kn = (form & HYC_GEMM_B_KN) != 0;
  if (count < 1 || count > 4 || M <= 0 || N <= 0 || N % BN != 0) return HYC_ERR_SHAPE;
  if (!aligned(D, 16) || (residual && !aligned(residual, 16))) return HYC_ERR_ALIGN;
  Operands ops = {};
  FourWeights four = {};
  for (int i = 0; i < count; ++i) {
    if (!A[i] || (!B[i] && !has_four(B4, i))) return HYC_ERR_NULL;
    if (K[i] <= 0 || K[i] % BK != 0) return HYC_ERR_SHAPE;
    if (has_four(B4, i)) {
      if (!four_takes(B4[i], M, b_is_kn ? N : K[i])) return HYC_ERR_UNSUPPORTED;
      if (!aligned(A[i], 16)) return HYC_ERR_ALIGN;
      ops.a[i] = {A[i], M, K[i]};
      four.w[i] = four_view(B4[i], b_is_kn ? N : K[i]);
      continue;
    }
    if (!aligned(A[i], 16) || !aligned(B[i], 16)) return HYC_ERR_ALIGN;
    ops.a[i] = {A[i], M, K[i]};
    ops.b[i] = b_is_kn ? Matrix{B[i], K[i], N} : Matrix{B[i], N, K[i]};
  }
  Params p = {};
  p.M = M; p.N = N; p.epi = EPI_STORE;
  p.fixed_order = (form & HYC_GEMM_FIXED_ORDER) != 0;
  p.K1 = K[0]; p.K2 = count > 1 ? K[1] : 0; p.K3 = count > 2 ? K[2] : 0; p.K4 = count > 3 ? K[3] : 0;
  p.residual = (const __nv_bfloat16*)residual;
  p.out0 = (__nv_bfloat16*)D;
  p.status = status;
  p.g_end0 = p.g_end1 = N;
  cudaStream_t st = (cudaStream_t)stream;
  const FourWeights* f4 = any_four(B4, count) ? &four : nullptr;
  return b_is_kn ? launch<EPI_STORE, 4, true>(ops, p, st, f4) : launch<EPI_STORE, 4, false>(ops, p, st, f4);
}
extern "C" HYC_API int hyc_gemm_segments_tcgen05(int count, const void* const* A, const void* const* B, const int* K, int M, int N,
                                                int form, const void* residual, void* D, int* status, void* stream) {
  return gemm_segments(count, A, B, nullptr, K, M, N, form, residual, D, status, stream);
}
extern "C" HYC_API int hyc_gemm_segments_nf4_tcgen05(int count, const void* const* A, const void* const* B, const hyc_nf4_weight* B4, const int* K,
                                                    int M, int N, int form, const void* residual, void* D, int* status, void* stream) {
  if (!B4) return HYC_ERR_NULL;
  return gemm_segments(count, A, B, B4, K, M, N, form, residual, D, status, stream);
}

static int gateup_fwd(
    const void* x, const void* wg, const void* wu, const hyc_nf4_weight* w4, int T, int H, int I,
    const void* xa1, const void* b1t, int64_t b1_ld_col, int64_t b1_ld_r,
    const void* xa2, const void* b2t, int64_t b2_ld_col, int64_t b2_ld_r,
    const void* s1, const void* s2, void* q1, void* q2, void* o, void* main1_or_null, void* main2_or_null,
    int q_bit, int* status, void* stream) {
  if (!x || (!w4 && (!wg || !wu)) || !xa1 || !b1t || !xa2 || !b2t || !s1 || !s2 || !q1 || !q2 || !o || !status) return HYC_ERR_NULL;
  if (q_bit != 2 && q_bit != 4 && q_bit != 8) return HYC_ERR_QBIT;
  if (T <= 0 || H <= 0 || I <= 0 || I % (BN / 2) != 0 || H % BK != 0) return HYC_ERR_SHAPE;
  if (w4 && (!four_takes(w4[0], T, H) || !four_takes(w4[1], T, H))) return HYC_ERR_UNSUPPORTED;
  const void* al[] = {x, wg, wu, xa1, xa2, q1, q2, o};
  for (const void* q : al) if (!aligned(q, 16)) return HYC_ERR_ALIGN;
  Operands ops = {};
  ops.a[0] = {x, T, H};
  ops.b[0] = {wg, I, H};
  ops.b[1] = {wu, I, H};
  FourWeights four = {};
  if (w4) { four.w[0] = four_view(w4[0], H); four.w[1] = four_view(w4[1], H); }
  const FourWeights* f4 = w4 ? &four : nullptr;
  Params p = {};
  p.M = T; p.N = I; p.K1 = H; p.K2 = 0; p.K3 = 0; p.epi = EPI_GATEUP; p.q_bit = q_bit;
  p.l0 = make_term(xa1, b1t, b1_ld_col, b1_ld_r);
  p.l1 = make_term(xa2, b2t, b2_ld_col, b2_ld_r);
  p.l2 = make_term(nullptr, nullptr, 0, 0);
  p.out0 = (__nv_bfloat16*)o;
  p.dbg1 = (__nv_bfloat16*)main1_or_null; p.dbg2 = (__nv_bfloat16*)main2_or_null;
  p.q1 = (uint8_t*)q1; p.q2 = (uint8_t*)q2;
  p.s1 = (const __nv_bfloat16*)s1; p.s2 = (const __nv_bfloat16*)s2;
  p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  p.g_end0 = p.g_end1 = I;
  if (q_bit == 2) return launch<EPI_GATEUP, 2, false>(ops, p, st, f4);
  if (q_bit == 4) return launch<EPI_GATEUP, 4, false>(ops, p, st, f4);
  return launch<EPI_GATEUP, 8, false>(ops, p, st, f4);
}

extern "C" HYC_API int hyc_mlp_gateup_fwd_tcgen05(
    const void* x, const void* wg, const void* wu,
    int T, int H, int I,
    const void* xa1, const void* b1t, int64_t b1_ld_col, int64_t b1_ld_r,
    const void* xa2, const void* b2t, int64_t b2_ld_col, int64_t b2_ld_r,
    const void* s1, const void* s2, void* q1, void* q2, void* o, void* main1_or_null, void* main2_or_null,
    int q_bit, int* status, void* stream) {
  return gateup_fwd(x, wg, wu, nullptr, T, H, I, xa1, b1t, b1_ld_col, b1_ld_r, xa2, b2t, b2_ld_col, b2_ld_r, s1, s2, q1, q2, o,
                    main1_or_null, main2_or_null, q_bit, status, stream);
}
extern "C" HYC_API int hyc_mlp_gateup_fwd_nf4_tcgen05(
    const void* x, const hyc_nf4_weight* gate_up,
    int T, int H, int I,
    const void* xa1, const void* b1t, int64_t b1_ld_col, int64_t b1_ld_r,
    const void* xa2, const void* b2t, int64_t b2_ld_col, int64_t b2_ld_r,
    const void* s1, const void* s2, void* q1, void* q2, void* o, void* main1_or_null, void* main2_or_null,
    int q_bit, int* status, void* stream) {
  if (!gate_up) return HYC_ERR_NULL;
  return gateup_fwd(x, nullptr, nullptr, gate_up, T, H, I, xa1, b1t, b1_ld_col, b1_ld_r, xa2, b2t, b2_ld_col, b2_ld_r, s1, s2, q1, q2, o,
                    main1_or_null, main2_or_null, q_bit, status, stream);
}

static int graddown_bwd(
    const void* g, const void* wd, const hyc_nf4_weight* w4, int T, int H, int I,
    const void* a_lora, const void* b_lora, int k_lora,
    const void* xa1, const void* b1t, int64_t b1_ld_col, int64_t b1_ld_r,
    const void* xa2, const void* b2t, int64_t b2_ld_col, int64_t b2_ld_r,
    const void* q1, const void* s1, const void* q2, const void* s2,
    const void* lora_gate, const void* lora_up, int64_t ld_lora,
    void* o, void* grad_gate, void* grad_up, int q_bit, int* status, void* stream) {
  if (!g || (!w4 && !wd) || !q1 || !s1 || !q2 || !s2 || !o || !grad_gate || !grad_up || !status) return HYC_ERR_NULL;
  const bool pre = lora_gate != nullptr || lora_up != nullptr;
  if (pre) {
    if (!lora_gate || !lora_up) return HYC_ERR_NULL;
    if (ld_lora < I || ld_lora % 8 != 0) return HYC_ERR_SHAPE;
    if (!aligned(lora_gate, 16) || !aligned(lora_up, 16)) return HYC_ERR_ALIGN;
  } else if (!xa1 || !b1t || !xa2 || !b2t) {
    return HYC_ERR_NULL;
  }
  if ((k_lora > 0) != (a_lora != nullptr && b_lora != nullptr)) return HYC_ERR_NULL;
  if (q_bit != 2 && q_bit != 4 && q_bit != 8) return HYC_ERR_QBIT;
  if (T <= 0 || H <= 0 || I <= 0 || I % BN != 0 || H % BK != 0 || k_lora < 0 || k_lora % BK != 0) return HYC_ERR_SHAPE;
  if (w4 && !four_takes(*w4, T, I)) return HYC_ERR_UNSUPPORTED;
  const void* al[] = {g, wd, q1, q2, o, grad_gate, grad_up};
  for (const void* q : al) if (!aligned(q, 16)) return HYC_ERR_ALIGN;
  if (!pre && (!aligned(xa1, 16) || !aligned(xa2, 16))) return HYC_ERR_ALIGN;
  if (a_lora && (!aligned(a_lora, 16) || !aligned(b_lora, 16))) return HYC_ERR_ALIGN;
  Operands ops = {};
  ops.a[0] = {g, T, H};
  ops.b[0] = {wd, H, I};      // [H, I] row-major: the K = H rows are the reduction dimension, so B is MN-major
  if (k_lora > 0) { ops.a[1] = {a_lora, T, k_lora}; ops.b[1] = {b_lora, k_lora, I}; }
  FourWeights four = {};
  if (w4) four.w[0] = four_view(*w4, I);
  const FourWeights* f4 = w4 ? &four : nullptr;
  Params p = {};
  p.M = T; p.N = I; p.K1 = H; p.K2 = k_lora; p.K3 = 0; p.epi = EPI_GRADDOWN; p.q_bit = q_bit;
  p.l0 = make_term(nullptr, nullptr, 0, 0);
  p.l1 = pre ? make_term(nullptr, nullptr, 0, 0) : make_term(xa1, b1t, b1_ld_col, b1_ld_r);
  p.l2 = pre ? make_term(nullptr, nullptr, 0, 0) : make_term(xa2, b2t, b2_ld_col, b2_ld_r);
  p.lpre1 = (const __nv_bfloat16*)lora_gate; p.lpre2 = (const __nv_bfloat16*)lora_up; p.ld_pre = ld_lora;
  p.out0 = (__nv_bfloat16*)o; p.out1 = (__nv_bfloat16*)grad_gate; p.out2 = (__nv_bfloat16*)grad_up;
  p.q1 = (uint8_t*)const_cast<void*>(q1); p.q2 = (uint8_t*)const_cast<void*>(q2);
  p.s1 = (const __nv_bfloat16*)s1; p.s2 = (const __nv_bfloat16*)s2;
  p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  p.g_end0 = p.g_end1 = I;
  if (q_bit == 2) return launch<EPI_GRADDOWN, 2, true>(ops, p, st, f4);
  if (q_bit == 4) return launch<EPI_GRADDOWN, 4, true>(ops, p, st, f4);
  return launch<EPI_GRADDOWN, 8, true>(ops, p, st, f4);
}

extern "C" HYC_API int hyc_mlp_graddown_bwd_tcgen05(
    const void* g, const void* wd,
    int T, int H, int I,
    const void* a_lora, const void* b_lora, int k_lora,
    const void* xa1, const void* b1t, int64_t b1_ld_col, int64_t b1_ld_r,
    const void* xa2, const void* b2t, int64_t b2_ld_col, int64_t b2_ld_r,
    const void* q1, const void* s1, const void* q2, const void* s2,
    const void* lora_gate, const void* lora_up, int64_t ld_lora,
    void* o, void* grad_gate, void* grad_up, int q_bit, int* status, void* stream) {
  return graddown_bwd(g, wd, nullptr, T, H, I, a_lora, b_lora, k_lora, xa1, b1t, b1_ld_col, b1_ld_r, xa2, b2t, b2_ld_col, b2_ld_r, q1, s1, q2, s2,
                      lora_gate, lora_up, ld_lora, o, grad_gate, grad_up, q_bit, status, stream);
}
extern "C" HYC_API int hyc_mlp_graddown_bwd_nf4_tcgen05(
    const void* g, const hyc_nf4_weight* down,
    int T, int H, int I,
    const void* a_lora, const void* b_lora, int k_lora,
    const void* xa1, const void* b1t, int64_t b1_ld_col, int64_t b1_ld_r,
    const void* xa2, const void* b2t, int64_t b2_ld_col, int64_t b2_ld_r,
    const void* q1, const void* s1, const void* q2, const void* s2,
    const void* lora_gate, const void* lora_up, int64_t ld_lora,
    void* o, void* grad_gate, void* grad_up, int q_bit, int* status, void* stream) {
  if (!down) return HYC_ERR_NULL;
  return graddown_bwd(g, nullptr, down, T, H, I, a_lora, b_lora, k_lora, xa1, b1t, b1_ld_col, b1_ld_r, xa2, b2t, b2_ld_col, b2_ld_r, q1, s1, q2, s2,
                      lora_gate, lora_up, ld_lora, o, grad_gate, grad_up, q_bit, status, stream);
}

// The LoRA projections of up to three weights on one x, with the saves of their main branches, in ONE launch: the tiles
// of all weights are dealt out together (separately every launch ends with a round of tiles that leaves SMs idle).
static int linears_lora_save(
    const void* x, int T, int K, int count, const void* const* w, const hyc_nf4_weight* w4, const int* n, const void* const* xa, const void* const* bt,
    const void* const* scale, void* const* q_out, void* const* y, int q_bit, int* status, void* stream) {
  if (!x || (!w && !w4) || !n || !xa || !bt || !scale || !q_out || !y || !status) return HYC_ERR_NULL;
  if (q_bit != 2 && q_bit != 4 && q_bit != 8) return HYC_ERR_QBIT;
  if (count < 1 || count > 3 || T <= 0 || K <= 0 || K % BK != 0) return HYC_ERR_SHAPE;
  if (!aligned(x, 16)) return HYC_ERR_ALIGN;
  int total = 0;
  Operands ops = {};
  FourWeights four = {};
  ops.a[0] = {x, T, K};
  for (int i = 0; i < count; ++i) {
    const bool coded = has_four(w4, i);
    if ((!coded && (!w || !w[i])) || !xa[i] || !bt[i] || !scale[i] || !q_out[i] || !y[i]) return HYC_ERR_NULL;
    if (n[i] <= 0 || n[i] % BN != 0) return HYC_ERR_SHAPE;
    if (coded && !four_takes(w4[i], T, K)) return HYC_ERR_UNSUPPORTED;
    if ((!coded && !aligned(w[i], 16)) || !aligned(xa[i], 16) || !aligned(q_out[i], 16) || !aligned(y[i], 16)) return HYC_ERR_ALIGN;
    if (coded) four.w[i] = four_view(w4[i], K);
    else ops.b[i] = {w[i], n[i], K};
    total += n[i];
  }
  Params p = {};
  p.M = T; p.N = total; p.K1 = K; p.epi = EPI_STORE; p.q_bit = q_bit;
  p.l0 = make_term(xa[0], bt[0], 16, 1);
  p.out0 = (__nv_bfloat16*)y[0]; p.q1 = (uint8_t*)q_out[0]; p.s1 = (const __nv_bfloat16*)scale[0];
  p.g_end0 = n[0];
  p.g_end1 = n[0] + (count > 1 ? n[1] : 0);
  Params::Group* g[2] = {&p.g1, &p.g2};
  for (int i = 1; i < count; ++i)
    *g[i - 1] = {(__nv_bfloat16*)y[i], (uint8_t*)q_out[i], (const __nv_bfloat16*)scale[i], make_term(xa[i], bt[i], 16, 1)};
  p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  const FourWeights* f4 = any_four(w4, count) ? &four : nullptr;
  if (q_bit == 2) return launch<EPI_STORE, 2, false>(ops, p, st, f4);
  if (q_bit == 4) return launch<EPI_STORE, 4, false>(ops, p, st, f4);
  return launch<EPI_STORE, 8, false>(ops, p, st, f4);
}

extern "C" HYC_API int hyc_linears_lora_save_fwd_tcgen05(
    const void* x, int T, int K, int count, const void* const* w, const int* n, const void* const* xa, const void* const* bt,
    const void* const* scale, void* const* q_out, void* const* y, int q_bit, int* status, void* stream) {
  return linears_lora_save(x, T, K, count, w, nullptr, n, xa, bt, scale, q_out, y, q_bit, status, stream);
}
extern "C" HYC_API int hyc_linears_lora_save_fwd_nf4_tcgen05(
    const void* x, int T, int K, int count, const void* const* w, const hyc_nf4_weight* w4, const int* n, const void* const* xa,
    const void* const* bt, const void* const* scale, void* const* q_out, void* const* y, int q_bit, int* status, void* stream) {
  if (!w4) return HYC_ERR_NULL;
  return linears_lora_save(x, T, K, count, w, w4, n, xa, bt, scale, q_out, y, q_bit, status, stream);
}

extern "C" HYC_API int hyc_linear_lora_save_fwd_tcgen05(
    const void* x, const void* w, int T, int K, int N,
    const void* xa, const void* bt, int64_t bt_ld_col, int64_t bt_ld_r,
    const void* scale, void* q_out, void* y, void* main_or_null, int q_bit, int* status, void* stream) {
  if (!x || !w || !scale || !q_out || !y || !status) return HYC_ERR_NULL;
  if ((xa != nullptr) != (bt != nullptr)) return HYC_ERR_NULL;
  if (q_bit != 2 && q_bit != 4 && q_bit != 8) return HYC_ERR_QBIT;
  if (T <= 0 || N <= 0 || K <= 0 || N % BN != 0 || K % BK != 0) return HYC_ERR_SHAPE;
  if (!aligned(x, 16) || !aligned(w, 16) || !aligned(y, 16) || !aligned(q_out, 16) || (xa && !aligned(xa, 16)) ||
      (main_or_null && !aligned(main_or_null, 16))) return HYC_ERR_ALIGN;
  Operands ops = {};
  ops.a[0] = {x, T, K};
  ops.b[0] = {w, N, K};
  Params p = {};
  p.M = T; p.N = N; p.K1 = K; p.K2 = 0; p.K3 = 0; p.epi = EPI_STORE; p.q_bit = q_bit;
  p.l0 = make_term(xa, bt, bt_ld_col, bt_ld_r);
  p.l1 = make_term(nullptr, nullptr, 0, 0);
  p.l2 = make_term(nullptr, nullptr, 0, 0);
  p.out0 = (__nv_bfloat16*)y;
  p.dbg1 = (__nv_bfloat16*)main_or_null;
  p.q1 = (uint8_t*)q_out;
  p.s1 = (const __nv_bfloat16*)scale;
  p.g_end0 = p.g_end1 = N;
  p.status = status;
  cudaStream_t st = (cudaStream_t)stream;
  if (q_bit == 2) return launch<EPI_STORE, 2, false>(ops, p, st);
  if (q_bit == 4) return launch<EPI_STORE, 4, false>(ops, p, st);
  return launch<EPI_STORE, 8, false>(ops, p, st);
}
