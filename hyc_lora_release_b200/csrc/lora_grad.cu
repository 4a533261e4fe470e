// LoRA-A gradient with the de-quantizer inside the contraction.
//
//   out[r, h] = sum_t gm[t, r] * x_hat[t, h],     x_hat = dequant(q, scale)
//
// The saved activation exists only as packed codes.  Each block owns 128 hidden columns and a
// chunk of tokens; per step it unpacks a 32-token x 128-column tile of codes into a bf16 tile in
// shared memory (one 32-column block of the packed layout per thread), and contracts it with the
// matching 32 x R tile of gm on the tensor cores (m16n8k16, fp32 accumulate; both operands are
// read from shared memory with transposing ldmatrix).  x_hat never goes to HBM: the kernel reads
// T*H*q/8 bytes of codes where the two-step version reads and writes 2*T*H bytes twice.
// Up to eight token chunks of the same columns are a cluster: their fp32 partials meet in distributed shared memory and
// are added up in the order of the chunks (narrow products of many tokens: several clusters, ga_shares).  The codes and gm rows of the next kGaAhead steps are on their way while a step is
// worked on: the kernel waits for memory (issue slots 0.1 without that, every step a full round trip).
// us, cold, with the second kernel that added the partials up before / now: 2048 tokens of 4096, 4 bits, one adapter 15.7 / 10.9,
// three 22.4 / 14.1; 128 tokens, 8 bits, two adapters 11.6 / 7.5; 8192 tokens, 8 bits, two 35.5 / 28.9.
#include "hyc_common.cuh"

namespace hyc {

constexpr int kGaCols = 128;      // hidden columns per block
constexpr int kGaStep = 32;       // tokens per step
constexpr int kGaMaxSplits = 8;   // token chunks = blocks of a cluster
constexpr int kGaAhead = 4;
constexpr int kGaMinSteps = 16;   // several clusters: steps per block at least
constexpr int kGaMaxR = 64;

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem_ptr) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(smem_ptr);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// de-quantize one 32-column block of one row into 32 bf16 (16 packed words), reference rounding
template <int QBIT> struct GaCodes { uint32_t w[QBIT]; };      // the packed bytes of a block
template <int QBIT>
__device__ __forceinline__ void load_codes32(const uint8_t* __restrict__ src, bool valid, GaCodes<QBIT>& c) {
#pragma unroll
  for (int i = 0; i < QBIT; ++i) c.w[i] = 0u;
  if (!valid) return;
  if constexpr (QBIT == 2) {
    const uint2 a = *reinterpret_cast<const uint2*>(src);
    c.w[0] = a.x; c.w[1] = a.y;
  } else {
#pragma unroll
    for (int i = 0; i < QBIT / 4; ++i) {
      const uint4 a = *reinterpret_cast<const uint4*>(src + 16 * i);
      c.w[4 * i] = a.x; c.w[4 * i + 1] = a.y; c.w[4 * i + 2] = a.z; c.w[4 * i + 3] = a.w;
    }
  }
}
template <int QBIT>
__device__ __forceinline__ void dequant_block32(const GaCodes<QBIT>& c, const uint32_t (&s2)[16], uint32_t (&out)[16]) {
  constexpr int EPP = 8 / QBIT, SLAB = 32 / EPP;
  constexpr uint32_t MASK = (1u << QBIT) - 1u, BM = MASK * 0x01010101u;
  const uint32_t (&w)[QBIT] = c.w;
  if constexpr (QBIT == 8) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {     // columns 2j, 2j+1 = bytes 2j, 2j+1
      const float f0 = (byte_to_magic_float(w[j >> 1], (2 * j) & 3) - 8388736.f) * bf16lo_to_f32(s2[j]);
      const float f1 = (byte_to_magic_float(w[j >> 1], ((2 * j) & 3) + 1) - 8388736.f) * bf16hi_to_f32(s2[j]);
      out[j] = pack_bf16x2_rn(f0, f1);
    }
  } else {
    constexpr uint32_t C1 = 0x4300u | (uint32_t)(1 << (QBIT - 1));
    const uint32_t c1 = C1 | (C1 << 16);
#pragma unroll
    for (int i = 0; i < EPP; ++i) {          // slab i: columns [i*SLAB, (i+1)*SLAB) = field i of bytes 0..SLAB-1
#pragma unroll
      for (int jj = 0; jj < SLAB / 2; ++jj) {
        const int byte0 = 2 * jj;            // bytes byte0, byte0+1 of the block
        const uint32_t f = (w[byte0 >> 2] >> (QBIT * i)) & BM;
        const uint32_t pr = __byte_perm(f, 0x43434343u, (byte0 & 2) ? 0x4342u : 0x4140u);
        __nv_bfloat162 t = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&pr), *reinterpret_cast<const __nv_bfloat162*>(&c1));
        const int j = (i * SLAB + byte0) >> 1;   // output pair index (columns 2j, 2j+1)
        t = __hmul2(t, *reinterpret_cast<const __nv_bfloat162*>(&s2[j]));
        out[j] = *reinterpret_cast<const uint32_t*>(&t);
      }
    }
  }
}

__device__ __forceinline__ uint32_t cluster_block_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_v4(const void* own, uint32_t rank) {      // the same variable in another block
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(own);
  uint32_t r;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r) : "memory");
  return v;
}

// four sums of a row of out, which may start at any element of a caller's buffer
__device__ __forceinline__ void store_sums(__nv_bfloat16* __restrict__ out, int64_t i, float4 s) {
  const uint2 w = make_uint2(pack_bf16x2_rn(s.x, s.y), pack_bf16x2_rn(s.z, s.w));
  if (aligned(out, 8)) {
    *reinterpret_cast<uint2*>(out + i) = w;
  } else {
    out[i] = __ushort_as_bfloat16((uint16_t)w.x); out[i + 1] = __ushort_as_bfloat16((uint16_t)(w.x >> 16));
    out[i + 2] = __ushort_as_bfloat16((uint16_t)w.y); out[i + 3] = __ushort_as_bfloat16((uint16_t)(w.y >> 16));
  }
}

// grid (hidden blocks, chunks, clusters), cluster (1, chunks).  RT = number of 16-row tiles of the LoRA dimension (R2 = 16 * RT).
// MANY: several clusters, each leaves its sums at ws, [cluster][R2][H] (a form of its own: the sums in memory cost the
// other one up to 10 % on 8-bit codes: 32768 tokens of 4096, three adapters, 97.9 us against 88.4)
template <int QBIT, int RT, bool MANY>
__global__ void __launch_bounds__(128)
lora_grad_a_kernel(const uint8_t* __restrict__ q, const __nv_bfloat16* __restrict__ scale,
                   const __nv_bfloat16* __restrict__ gm, int64_t ldg, int T, int H, int chunk, __nv_bfloat16* __restrict__ out,
                   float* __restrict__ ws) {
  pdl_wait();
  constexpr int R2 = 16 * RT, PIECES = kGaStep * (R2 / 8), PPT = (PIECES + 127) / 128;      // 16-byte pieces of a gm tile, per thread
  constexpr int X_LD = kGaCols + 8, G_LD = R2 + 8;
  // the tiles of two steps; after the last one the partials take their place
  constexpr int X_BYTES = 2 * kGaStep * X_LD * 2, TILE_BYTES = X_BYTES + 2 * kGaStep * G_LD * 2, PART_BYTES = R2 * (kGaCols + 4) * 4;
  __shared__ __align__(16) uint8_t s_raw[TILE_BYTES > PART_BYTES ? TILE_BYTES : PART_BYTES];
  auto xs = reinterpret_cast<__nv_bfloat16 (*)[kGaStep][X_LD]>(s_raw);
  auto gs = reinterpret_cast<__nv_bfloat16 (*)[kGaStep][G_LD]>(s_raw + X_BYTES);
  auto part = reinterpret_cast<float (*)[kGaCols + 4]>(s_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h0 = blockIdx.x * kGaCols;
  const int t_begin = (MANY ? blockIdx.z * gridDim.y + blockIdx.y : blockIdx.y) * chunk;
  const int t_end = min(T, t_begin + chunk);
  const int64_t qld = (int64_t)H * QBIT / 8;

  // this thread de-quantizes block `blk` (32 columns) of row `lrow` of every step
  const int lrow = tid >> 2, blk = tid & 3;
  const uint8_t* qp = q + (int64_t)(t_begin + lrow) * qld + (int64_t)(h0 + 32 * blk) * QBIT / 8;
  GaCodes<QBIT> codes[kGaAhead];
  uint4 gmv[kGaAhead][PPT];
  auto fetch = [&](int t0, int slot) {
    load_codes32<QBIT>(qp + (int64_t)(t0 - t_begin) * qld, t0 + lrow < t_end, codes[slot]);
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      const int p = tid + 128 * i, r = p / (R2 / 8), c = p % (R2 / 8);
      gmv[slot][i] = make_uint4(0u, 0u, 0u, 0u);
      if (p < PIECES && t0 + r < t_end) gmv[slot][i] = *reinterpret_cast<const uint4*>(gm + (int64_t)(t0 + r) * ldg + 8 * c);
    }
  };
#pragma unroll
  for (int i = 0; i < kGaAhead; ++i) fetch(t_begin + kGaStep * i, i);
  uint32_t s2[16];
  {
    const uint4* sp = reinterpret_cast<const uint4*>(scale + h0 + 32 * blk);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const uint4 v = sp[i]; s2[4 * i] = v.x; s2[4 * i + 1] = v.y; s2[4 * i + 2] = v.z; s2[4 * i + 3] = v.w; }
  }
  float acc[RT][4][4];
#pragma unroll
  for (int m = 0; m < RT; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;

  for (int tb = t_begin; tb < t_end; tb += kGaStep * kGaAhead) {
#pragma unroll
    for (int u = 0; u < kGaAhead; ++u) {
      const int t0 = tb + kGaStep * u, buf = u & 1;
      if (t0 >= t_end) break;
      uint32_t xv[16];
      dequant_block32<QBIT>(codes[u], s2, xv);
      if (t0 + lrow >= t_end) {
#pragma unroll
        for (int j = 0; j < 16; ++j) xv[j] = 0u;
      }
      uint4* xdst = reinterpret_cast<uint4*>(&xs[buf][lrow][32 * blk]);
#pragma unroll
      for (int i = 0; i < 4; ++i) xdst[i] = make_uint4(xv[4 * i], xv[4 * i + 1], xv[4 * i + 2], xv[4 * i + 3]);
#pragma unroll
      for (int i = 0; i < PPT; ++i) {
        const int p = tid + 128 * i;
        if (p < PIECES) *reinterpret_cast<uint4*>(&gs[buf][p / (R2 / 8)][8 * (p % (R2 / 8))]) = gmv[u][i];
      }
      fetch(t0 + kGaStep * kGaAhead, u);
      __syncthreads();      // (one barrier per step: the tile written next was read a step ago)
#pragma unroll
      for (int kk = 0; kk < kGaStep / 16; ++kk) {
        const int k0 = 16 * kk;
        uint32_t a[RT][4];
#pragma unroll
        for (int m = 0; m < RT; ++m)
          ldmatrix_x4_trans(a[m], &gs[buf][k0 + (lane & 7) + ((lane >> 4) & 1) * 8][16 * m + ((lane >> 3) & 1) * 8]);
#pragma unroll
        for (int np = 0; np < 2; ++np) {     // two 8-column tiles per ldmatrix
          uint32_t b[4];
          ldmatrix_x4_trans(b, &xs[buf][k0 + (lane & 7) + ((lane >> 3) & 1) * 8][32 * warp + 16 * np + ((lane >> 4) & 1) * 8]);
#pragma unroll
          for (int m = 0; m < RT; ++m) {
            mma16816(acc[m][2 * np], a[m], b[0], b[1]);
            mma16816(acc[m][2 * np + 1], a[m], b[2], b[3]);
          }
        }
      }
    }
  }
  __syncthreads();
  const int g = lane >> 2, tq = lane & 3;
#pragma unroll
  for (int m = 0; m < RT; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int h = 32 * warp + 8 * n + 2 * tq;
      *reinterpret_cast<float2*>(&part[16 * m + g][h]) = make_float2(acc[m][n][0], acc[m][n][1]);
      *reinterpret_cast<float2*>(&part[16 * m + g + 8][h]) = make_float2(acc[m][n][2], acc[m][n][3]);
    }
  // every block of the cluster adds up its share of the rows
  const int splits = (int)gridDim.y;
  if (splits > 1) cluster_barrier(); else __syncthreads();
  for (int r = (splits > 1 ? (int)cluster_block_rank() : 0) * 4 + warp; r < R2; r += 4 * splits) {
    const int h = 4 * lane;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < splits; ++k) {
      const float4 v = splits > 1 ? ld_cluster_v4(&part[r][h], (uint32_t)k) : *reinterpret_cast<const float4*>(&part[r][h]);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const int64_t i = (int64_t)r * H + h0 + h;
    if (MANY) *reinterpret_cast<float4*>(ws + (int64_t)blockIdx.z * R2 * H + i) = s;
    else store_sums(out, i, s);
  }
  if (splits > 1) cluster_barrier();      // nobody leaves while its partials may be read
}

// the clusters' sums, in their order (n = R2 * H)
__global__ void __launch_bounds__(128)
lora_grad_a_sum_kernel(const float* __restrict__ ws, int clusters, int64_t n, __nv_bfloat16* __restrict__ out) {
  pdl_wait();
  const int64_t i = 4 * ((int64_t)blockIdx.x * 128 + threadIdx.x);      // (n is a multiple of 2048)
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < clusters; ++k) {
    const float4 v = *reinterpret_cast<const float4*>(ws + k * n + i);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  store_sums(out, i, s);
}

// How the tokens are shared: whole steps each, eight blocks at most per cluster.  One cluster per 128 columns where these fill
// the GPU or the tokens are few; narrower products of many tokens take several (four blocks per SM, 512 tokens per block at
// least), which meet in a workspace.  us, one cluster / several, 4 bits, two adapters: 32768 tokens of 1024 columns 54.8 / 21.8, of
// 2048 65.5 / 34.6, of 128 51.2 / 12.5; 8192 of 1024 16.8 / 13.7 (256 tokens per block: 10.8, but 4096 of 1024 then take 9.5
// against 8.9 of one cluster).
struct GaShares { int clusters, blocks, chunk; };
static GaShares ga_shares(int T, int H) {
  const int steps = (T + kGaStep - 1) / kGaStep, one = H / kGaCols * kGaMaxSplits;
  int clusters = 1;
  if (one < num_sms()) {
    const int room = 4 * num_sms() / one, wanted = steps / (kGaMaxSplits * kGaMinSteps);
    clusters = wanted < 1 ? 1 : (wanted < room ? wanted : room);
  }
  const int shares = clusters * kGaMaxSplits, chunk = (steps + shares - 1) / shares * kGaStep;
  return {clusters, clusters > 1 ? kGaMaxSplits : (T + chunk - 1) / chunk, chunk};
}

}  // namespace hyc

using namespace hyc;

extern "C" HYC_API size_t hyc_lora_grad_a_workspace_bytes(int T, int H, int R2) {
  if (T <= 0 || H < kGaCols || R2 <= 0) return 0;
  const GaShares g = ga_shares(T, H);
  return g.clusters > 1 ? (size_t)g.clusters * (size_t)R2 * (size_t)H * sizeof(float) : 0;
}

template <int QBIT, int RT>
static int launch_ga(const void* q, const void* scale, const void* gm, int64_t ldg, int T, int H, void* out, void* workspace, cudaStream_t st) {
  const GaShares g = ga_shares(T, H);
  float* ws = g.clusters > 1 ? (float*)workspace : nullptr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(H / kGaCols), (unsigned)g.blocks, (unsigned)g.clusters);
  cfg.blockDim = dim3(128);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = (unsigned)g.blocks; at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = g.blocks > 1 ? 2 : 1;
  (void)cudaLaunchKernelEx(&cfg, ws != nullptr ? lora_grad_a_kernel<QBIT, RT, true> : lora_grad_a_kernel<QBIT, RT, false>, (const uint8_t*)q, (const __nv_bfloat16*)scale, (const __nv_bfloat16*)gm, ldg, T, H,
                           g.chunk, (__nv_bfloat16*)out, ws);
  HYC_CHECK_LAUNCH();
  if (ws != nullptr) {
    const int64_t n = (int64_t)16 * RT * H;
    launch_pdl(lora_grad_a_sum_kernel, dim3((unsigned)(n / 512)), dim3(128), 0, st, (const float*)ws, g.clusters, n, (__nv_bfloat16*)out);
    HYC_CHECK_LAUNCH();
  }
  return HYC_OK;
}

extern "C" HYC_API int hyc_lora_grad_a_dequant(const void* q, const void* scale, const void* gm, int64_t ldg, int R2,
                                               int T, int H, int q_bit, void* out, void* workspace, size_t workspace_bytes,
                                               void* stream) {
  if (!q || !scale || !gm || !out) return HYC_ERR_NULL;
  if (q_bit != 2 && q_bit != 4 && q_bit != 8) return HYC_ERR_QBIT;
  if (T <= 0 || H <= 0 || H % kGaCols != 0 || R2 <= 0 || R2 % 16 != 0 || R2 > kGaMaxR || ldg < R2) return HYC_ERR_SHAPE;
  if (!aligned(q, 16) || !aligned(scale, 16) || !aligned(gm, 16) || ldg % 8 != 0 || !aligned(workspace, 16)) return HYC_ERR_ALIGN;
  const size_t need = hyc_lora_grad_a_workspace_bytes(T, H, R2);
  if (need > 0 && !workspace) return HYC_ERR_NULL;
  if (workspace_bytes < need) return HYC_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
#define GA(QB, RT) return launch_ga<QB, RT>(q, scale, gm, ldg, T, H, out, workspace, st)
#define GAQ(QB) switch (R2 / 16) { case 1: GA(QB, 1); case 2: GA(QB, 2); case 3: GA(QB, 3); default: GA(QB, 4); }
  if (q_bit == 2) { GAQ(2) }
  if (q_bit == 4) { GAQ(4) }
  GAQ(8)
#undef GAQ
#undef GA
}
