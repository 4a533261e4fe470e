// Rank-16 products with a large operand X [T, N]:  Y = X W (W [N, 16], up to three of them) and Z = X^T xa (xa [T, 16]),
// both from ONE read of X, for up to three X in one launch.
//
// The backward pass needs both forms of every gradient (g B for the input's gradient, g^T xa for B's).  Each is bound by
// reading X; as library calls they read it twice, and each call costs the host 10 us.  One call for grad_gate, grad_up and
// hadamard of 2048 tokens (three X of [2048, 11008], 135 MB from HBM): 39 us with its sums, 33 of them the first kernel's,
// which is then at 52 % of the DRAM rate (issue slots 7 %: it waits for its tiles).
//
// A CTA owns a region of R x C tiles of 128 x 128 of one X.  A tile arrives by TMA (128-byte swizzle) and is the A operand
// of both products as it lies: rows x K for Y (K = its columns), transposed for Z (K = its rows); W and xa come once per
// region as 32-byte-swizzled [128][16] blocks, an MN-major B operand of N = 16.  All R x n_w accumulators of Y and all C
// of Z stay in tensor memory (16 columns each) and leave once, as fp32 partials that a second, small kernel adds up in
// a fixed order and converts: Y over the column regions, Z over the row regions.
// On mma.sync the same plan was bound by that pipe (93 % busy, about 256 MAC per cycle and SM): three X of [8192, 14336]
// 162 us = 4.3 TB/s.
#include "tc_common.cuh"

namespace hyc {
namespace sk {

using namespace tc;

constexpr int TILE = 128, X_BYTES = TILE * TILE * 2, AUX_BYTES = TILE * 32;
constexpr int MAXJ = 3, RING = 5, AUX_SLOTS = 14;      // R + n_w C <= AUX_SLOTS
constexpr int SK_THREADS = 64 + 128;
constexpr int AUX_AT = RING * X_BYTES, BARS_AT = AUX_AT + AUX_SLOTS * AUX_BYTES;
constexpr int SK_SMEM = 1024 + BARS_AT + 256;

struct JobMaps { CUtensorMap x, w[MAXJ], xa; };
struct Job {
  __nv_bfloat16* y[MAXJ];
  __nv_bfloat16* z;
  float* yp;                      // [n_w][column regions][T][16]
  float* zp;                      // [row regions][n][16]
  int64_t ld_y;
  int n, n_w, y_pad, z_transposed, first_region, col_regions;
};
struct Args {
  JobMaps maps[MAXJ];
  Job job[MAXJ];
  int count, T, R, C, row_regions;
  int* status;
};

__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                 "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// X tile (two boxes of 64 columns) for K step kk of 16: rows x K, and columns x K
__device__ __forceinline__ uint64_t x_rows(uint32_t tile, int kk) {
  return make_desc(tile + (uint32_t)((kk >> 2) * (X_BYTES / 2) + (kk & 3) * 32), 16, 1024);
}
__device__ __forceinline__ uint64_t x_cols(uint32_t tile, int kk) { return make_desc(tile + (uint32_t)(kk * 2048), X_BYTES / 2, 1024); }
// [128][16] block, 32-byte swizzle, N contiguous: groups of eight K rows are 256 bytes apart
__device__ __forceinline__ uint64_t aux_desc(uint32_t block, int kk) {
  uint64_t d = 0;
  d |= (uint64_t)(((block + (uint32_t)kk * 512u) & 0x3ffffu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(256 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)6 << 61;
  return d;
}
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((16u >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
constexpr uint32_t kAMn = 1u << 15;

__global__ void __launch_bounds__(SK_THREADS, 1)
skinny_kernel(const __grid_constant__ Args a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_shared(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + BARS_AT);
  uint64_t *full = bars, *empty = bars + RING, *aux_full = bars + 2 * RING, *acc_full = aux_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  int ji = 0;
  while (ji + 1 < a.count && (int)blockIdx.x >= a.job[ji + 1].first_region) ++ji;
  const Job& j = a.job[ji];
  const JobMaps& m = a.maps[ji];
  const int region = (int)blockIdx.x - j.first_region, cr = region % j.col_regions, rr = region / j.col_regions;
  const int row0 = rr * a.R * TILE, col0 = cr * a.C * TILE;
  const int nr = min(a.R, (a.T - row0 + TILE - 1) / TILE), nc = min(a.C, (j.n - col0 + TILE - 1) / TILE);
  const int n_w = j.n_w;
  const bool cz = j.z != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RING; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(aux_full, 1);
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();      // before tensor memory is taken: see launch_pdl
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t ring = smem_u32(smem), aux = ring + AUX_AT;
  // xa blocks first, then W blocks [column tile][w]; accumulators: Y [row tile][w], then Z [column tile]
  const uint32_t w_at = aux + (uint32_t)((cz ? nr : 0) * AUX_BYTES), z_at = tmem + (uint32_t)(nr * n_w * 16);

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(aux_full, (uint32_t)(((cz ? nr : 0) + nc * n_w) * AUX_BYTES));
      if (cz)
        for (int r = 0; r < nr; ++r) tma_load_2d<false>(aux + r * AUX_BYTES, &m.xa, smem_u32(aux_full), 0, row0 + r * TILE);
      for (int c = 0; c < nc; ++c)
        for (int w = 0; w < n_w; ++w) tma_load_2d<false>(w_at + (c * n_w + w) * AUX_BYTES, &m.w[w], smem_u32(aux_full), 0, col0 + c * TILE);
    }
    __syncwarp();
    int slot = 0;
    uint32_t phase = 0;
    for (int t = 0; t < nr * nc; ++t) {
      if (!mbar_wait_warp(&empty[slot], phase ^ 1u, abort_flag)) {
        if (lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(a.status, ST_TIMEOUT_PRODUCER); }
        break;
      }
      if (elect_one()) {
        const uint32_t dst = ring + (uint32_t)slot * X_BYTES;
        const int x0 = col0 + (t % nc) * TILE, y0 = row0 + (t / nc) * TILE;
        mbar_expect_tx(&full[slot], X_BYTES);
        tma_load_2d<false>(dst, &m.x, smem_u32(&full[slot]), x0, y0);
        tma_load_2d<false>(dst + X_BYTES / 2, &m.x, smem_u32(&full[slot]), x0 + 64, y0);
      }
      __syncwarp();
      if (++slot == RING) { slot = 0; phase ^= 1u; }
    }
  } else if (warp == 1) {
    int slot = 0;
    uint32_t phase = 0;
    bool ok = mbar_wait_warp(aux_full, 0, abort_flag);
    for (int t = 0; t < nr * nc && ok; ++t) {
      ok = mbar_wait_warp(&full[slot], phase, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const int r = t / nc, c = t % nc;
      const uint32_t x = ring + (uint32_t)slot * X_BYTES;
      if (elect_one()) {
        for (int w = 0; w < n_w; ++w) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma<false>(tmem + (uint32_t)((r * n_w + w) * 16), x_rows(x, kk), aux_desc(w_at + (c * n_w + w) * AUX_BYTES, kk), kIdesc, (c > 0 || kk > 0) ? 1u : 0u);
        }
        if (cz) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            tc_mma<false>(z_at + (uint32_t)(c * 16), x_cols(x, kk), aux_desc(aux + r * AUX_BYTES, kk), kIdesc | kAMn, (r > 0 || kk > 0) ? 1u : 0u);
        }
        tc_commit<false>(&empty[slot]);
        if (t + 1 == nr * nc) tc_commit<false>(acc_full);
      }
      __syncwarp();
      if (++slot == RING) { slot = 0; phase ^= 1u; }
    }
    if (!ok && lane == 0 && !*abort_flag) { *abort_flag = 1; atomicExch(a.status, ST_TIMEOUT_MMA); }
  } else {
    const int quad = warp & 3, i = quad * 32 + lane;
    bool ok = mbar_wait(acc_full, 0, abort_flag);
    if (!ok && !*abort_flag) { *abort_flag = 1; atomicExch(a.status, ST_TIMEOUT_EPILOGUE); }
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    if (ok) {
      const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
      const int ny = nr * n_w, total = ny + (cz ? nc : 0);
#pragma unroll 1
      for (int k = 0; k < total; ++k) {
        uint32_t v[16];
        tc_ld16(tmem + t_lane + (uint32_t)(k * 16), v);
        const bool is_y = k < ny;
        const int64_t at = is_y ? row0 + (k / max(n_w, 1)) * TILE + i : col0 + (k - ny) * TILE + i;
        float* dst = is_y ? j.yp + ((int64_t)(k % max(n_w, 1)) * j.col_regions + cr) * a.T * 16 : j.zp + (int64_t)rr * j.n * 16;
        if (at < (is_y ? a.T : j.n)) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            *reinterpret_cast<uint4*>(dst + at * 16 + 4 * e) = make_uint4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Sums of the partials, four values of the result at a time: partials k, k + 8, ... first, then these eight in order.
struct SumAt {
  const float* p;                 // its first partial
  int64_t e, stride;
  int w, parts;
  bool is_y;
  __device__ __forceinline__ SumAt(const Args& a, const Job& j, int64_t i, int64_t ny) {
    is_y = i < ny;
    w = is_y ? (int)(i / ((int64_t)a.T * 4)) : 0;
    e = is_y ? i - (int64_t)w * a.T * 4 : i - ny;
    stride = is_y ? (int64_t)a.T * 16 : (int64_t)j.n * 16;
    parts = is_y ? j.col_regions : a.row_regions;
    p = (is_y ? j.yp + (int64_t)w * j.col_regions * a.T * 16 : j.zp) + e * 4;
  }
};
__device__ __forceinline__ void add4(float4& s, const float4& v) { s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
__device__ __forceinline__ void sum_store(const Job& j, const SumAt& t, const float4& s) {
  const int64_t at = t.e >> 2;
  const int r = 4 * (int)(t.e & 3);
  const uint2 out = make_uint2(pack_bf16x2_rn(s.x, s.y), pack_bf16x2_rn(s.z, s.w));
  if (t.is_y) {
    __nv_bfloat16* y = j.y[t.w] + at * j.ld_y + r;
    *reinterpret_cast<uint2*>(y) = out;
    // zero columns behind the last product of the job (it rides a GEMM as part of a K block of 64)
    if (t.w == j.n_w - 1)
      for (int c = 0; c < j.y_pad; c += 16) *reinterpret_cast<uint2*>(y + 16 + c) = make_uint2(0u, 0u);
  } else if (j.z_transposed) {
    const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) j.z[(int64_t)(r + c) * j.n + at] = __float2bfloat16_rn(v[c]);
  } else {
    *reinterpret_cast<uint2*>(j.z + at * 16 + r) = out;
  }
}

// Many partials: the eight warps of a block take every eighth partial of 32 results each and meet in shared memory
// (one thread adding 43 of them one after the other took 5 us at 2048 rows).
__global__ void __launch_bounds__(256)
sum_kernel(const __grid_constant__ Args a) {
  pdl_wait();
  __shared__ float4 s_part[8][32];
  const Job& j = a.job[blockIdx.y];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ny = (int64_t)j.n_w * a.T * 4, nz = j.z != nullptr ? (int64_t)j.n * 4 : 0;
  for (int64_t base = (int64_t)blockIdx.x * 32; base < ny + nz; base += (int64_t)gridDim.x * 32) {
    const bool valid = base + lane < ny + nz;
    const SumAt t(a, j, base + lane, ny);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) {
#pragma unroll 4
      for (int k = warp; k < t.parts; k += 8) add4(s, __ldcg(reinterpret_cast<const float4*>(t.p + k * t.stride)));
    }
    s_part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && valid) {
#pragma unroll
      for (int k = 1; k < 8; ++k) add4(s, s_part[k][lane]);
      sum_store(j, t, s);
    }
    __syncthreads();
  }
}

// Up to sixteen partials: a thread has them all on their way at once.  Taken where that makes a block per SM: three X of [2048, 11008] 10.2 ->
// 6.0 us (the other way it is 4896 blocks of a barrier and a few loads each); one X of [2048, 4096], 96 blocks, would take 5.1 for 4.4.
constexpr int kFewParts = 16;
__global__ void __launch_bounds__(256)
sum_few_kernel(const __grid_constant__ Args a) {
  pdl_wait();
  const Job& j = a.job[blockIdx.y];
  const int64_t ny = (int64_t)j.n_w * a.T * 4, nz = j.z != nullptr ? (int64_t)j.n * 4 : 0;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= ny + nz) return;
  const SumAt t(a, j, i, ny);
  float4 v[kFewParts];
#pragma unroll
  for (int k = 0; k < kFewParts; ++k) {
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < t.parts) v[k] = __ldcg(reinterpret_cast<const float4*>(t.p + k * t.stride));
  }
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float4 pair = v[k];
    add4(pair, v[k + 8]);
    if (k == 0) s = pair;
    else add4(s, pair);
  }
  sum_store(j, t, s);
}

// row-major bf16 [rows, cols] with a row stride of its own; box = box_cols x 128 rows
static bool map_2d(CUtensorMap* m, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_cols, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)TILE};
  cuuint32_t estr[2] = {1u, 1u};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// R x C tiles of a region (one CTA per SM at a time): fewest tiles on the busiest SM, filling and leaving the pipeline
// counted as six tiles, then the fewest partials
struct Plan { int R, C, regions; };
static Plan make_plan(int count, const hyc_skinny_job* jobs, int T) {
  const int tr = (T + TILE - 1) / TILE, sms = num_sms();
  int n_w = 0, widest = 0;
  for (int i = 0; i < count; ++i) {
    n_w = jobs[i].n_w > n_w ? jobs[i].n_w : n_w;
    const int tc = (jobs[i].n + TILE - 1) / TILE;
    widest = tc > widest ? tc : widest;
  }
  Plan best = {1, 1, 0};
  int64_t best_cost = INT64_MAX;
  for (int R = 1; R <= tr && R < AUX_SLOTS; ++R) {
    for (int C = 1; C <= widest && R + n_w * C <= AUX_SLOTS && R * n_w + C <= 32; ++C) {
      int regions = 0;
      const int rows = (tr + R - 1) / R;
      for (int i = 0; i < count; ++i) regions += rows * (((jobs[i].n + TILE - 1) / TILE + C - 1) / C);
      const int64_t waves = (regions + sms - 1) / sms;
      const int64_t cost = waves * (R * C + 6) * 4096 + regions * (R + C);
      if (cost < best_cost) { best_cost = cost; best = {R, C, regions}; }
    }
  }
  return best;
}
static size_t ws_floats(int count, const hyc_skinny_job* jobs, int T, const Plan& p) {
  const int tr = (T + TILE - 1) / TILE, rows = (tr + p.R - 1) / p.R;
  size_t f = 0;
  for (int i = 0; i < count; ++i) {
    const int cols = ((jobs[i].n + TILE - 1) / TILE + p.C - 1) / p.C;
    f += (size_t)jobs[i].n_w * cols * T * 16 + (jobs[i].z ? (size_t)rows * jobs[i].n * 16 : 0);
  }
  return f;
}

}  // namespace sk
}  // namespace hyc

using namespace hyc;
using namespace hyc::sk;

extern "C" HYC_API size_t hyc_skinny_workspace_bytes(int count, const hyc_skinny_job* jobs, int T) {
  if (count < 1 || count > MAXJ || !jobs || T <= 0) return 0;
  return ws_floats(count, jobs, T, make_plan(count, jobs, T)) * 4;
}

extern "C" HYC_API int hyc_skinny_products(int count, const hyc_skinny_job* jobs, int T, void* workspace, size_t workspace_bytes, int* status,
                                           void* stream) {
  if (!jobs || !workspace || !status) return HYC_ERR_NULL;
  if (count < 1 || count > MAXJ || T <= 0) return HYC_ERR_SHAPE;
  for (int i = 0; i < count; ++i) {
    const hyc_skinny_job& s = jobs[i];
    if (!s.x || (s.xa != nullptr) != (s.z != nullptr)) return HYC_ERR_NULL;
    if (s.n <= 0 || s.n % 8 != 0 || s.n_w < 0 || s.n_w > MAXJ || (s.n_w == 0 && !s.z) || s.ldx < s.n || s.y_pad < 0 || s.y_pad % 16 != 0) return HYC_ERR_SHAPE;
    if (!aligned(s.x, 16) || s.ldx % 8 != 0 || (s.xa && (!aligned(s.xa, 16) || s.ld_xa % 8 != 0)) || (s.z && !aligned(s.z, 8))) return HYC_ERR_ALIGN;
    for (int w = 0; w < s.n_w; ++w) {
      if (!s.w[w] || !s.y[w]) return HYC_ERR_NULL;
      if (!aligned(s.w[w], 16) || s.ld_w % 8 != 0 || !aligned(s.y[w], 8) || s.ld_y % 4 != 0) return HYC_ERR_ALIGN;
    }
  }
  const Plan plan = make_plan(count, jobs, T);
  if (workspace_bytes < ws_floats(count, jobs, T, plan) * 4) return HYC_ERR_WORKSPACE;
  if (!aligned(workspace, 16)) return HYC_ERR_ALIGN;
  Args a = {};
  a.count = count; a.T = T; a.R = plan.R; a.C = plan.C; a.status = status;
  a.row_regions = ((T + TILE - 1) / TILE + plan.R - 1) / plan.R;
  float* ws = (float*)workspace;
  int64_t most = 0;
  int first = 0;
  for (int i = 0; i < count; ++i) {
    const hyc_skinny_job& s = jobs[i];
    Job& j = a.job[i];
    JobMaps& m = a.maps[i];
    bool ok = map_2d(&m.x, s.x, T, s.n, s.ldx, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    for (int w = 0; w < s.n_w; ++w) {
      ok = ok && map_2d(&m.w[w], s.w[w], s.n, 16, s.ld_w, 16, CU_TENSOR_MAP_SWIZZLE_32B);
      j.y[w] = (__nv_bfloat16*)s.y[w];
    }
    if (s.xa) ok = ok && map_2d(&m.xa, s.xa, T, 16, s.ld_xa, 16, CU_TENSOR_MAP_SWIZZLE_32B);
    if (!ok) return HYC_ERR_UNSUPPORTED;
    j.z = (__nv_bfloat16*)s.z;
    j.ld_y = s.ld_y;
    j.n = s.n; j.n_w = s.n_w; j.y_pad = s.y_pad; j.z_transposed = s.z_transposed;
    j.first_region = first;
    j.col_regions = ((s.n + TILE - 1) / TILE + plan.C - 1) / plan.C;
    first += a.row_regions * j.col_regions;
    j.yp = ws; ws += (size_t)j.n_w * j.col_regions * T * 16;
    j.zp = ws; if (j.z) ws += (size_t)a.row_regions * j.n * 16;
    const int64_t outs = (int64_t)j.n_w * T * 4 + (j.z ? (int64_t)j.n * 4 : 0);
    most = outs > most ? outs : most;
  }
  static bool attr[64] = {false};
  const int slot = current_device_slot();
  if (slot < 0 || !attr[slot]) {
    if (cudaFuncSetAttribute(skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SK_SMEM) != cudaSuccess) {
      hyc_set_last_cuda_error((int)cudaGetLastError());
      return HYC_ERR_LAUNCH;
    }
    if (slot >= 0) attr[slot] = true;
  }
  cudaStream_t st = (cudaStream_t)stream;
  launch_pdl(skinny_kernel, dim3((unsigned)first), dim3(SK_THREADS), SK_SMEM, st, a);
  HYC_CHECK_LAUNCH();
  int parts = a.row_regions;
  for (int i = 0; i < count; ++i) parts = a.job[i].n_w > 0 && a.job[i].col_regions > parts ? a.job[i].col_regions : parts;
  const int64_t few = (most + 255) / 256;
  if (parts <= kFewParts && few * count >= num_sms()) {
    launch_pdl(sum_few_kernel, dim3((unsigned)few, count), dim3(256), 0, st, a);
  } else {
    const int64_t grid = (most + 31) / 32;
    launch_pdl(sum_kernel, dim3((unsigned)(grid < 4096 ? grid : 4096), count), dim3(256), 0, st, a);
  }
  HYC_CHECK_LAUNCH();
  return HYC_OK;
}
