// Stage 3b for fp32 inputs: block-sparse causal flash-attention forward on the CUDA cores, register-tiled.
//
// Same math as pbs_attn_simt.cu (pbs_attn/src/kernels/permuted_block_sparse_attention.py:7-90,241-311): fp32
// scores scaled by 1/sqrt(D), key visible iff its original position <= the query's, online softmax in base 2,
// fp32 accumulators.  There is no fp32 tensor-core path, so the bound is the fp32 FMA rate: 4*D FLOP per
// (query, key) of the kept blocks.  One CTA = 32 query rows; a step = 64 keys of one kept block, brought in by
// cp.async.  Loads are hidden by the other CTAs of the SM (four at head_dim 64, two at 128), not by a second buffer: with one at
// head_dim 64 there were two CTAs a SM, 4 heads x 8192 tokens 1033 us against 927.
// 128 threads as 8 x 16: a thread owns 4 rows x 4 keys of S and 4 rows x D/16 columns of O, so 32 packed FMA pairs feed
// on 8 shared-memory reads of 16 bytes, and the 16 lanes that share rows reduce them by shuffles and pass P through
// shared memory without a block-wide barrier.  The products of two neighbouring head-dim elements go into two partial
// sums (packed fp32 pairs), which are added at the end of the row.
// A step takes 2 to 4 us, so few query tiles leave the GPU waiting for the longest row: then a cluster of 2, 4 or 8 CTAs shares a query
// tile's steps and puts O together through distributed shared memory.  While the GPU has places for all CTAs (the line: 4 heads x
// 2048 tokens with 1 / 4 / 8 CTAs a tile 130 / 83 / 89 us; 8 heads of 128, whose tiles alone take all places, 257 with 1, 282 with 4);
// 4 heads of 64: 300 tokens 23 -> 18 us, 1000 tokens 58 -> 36, 2048 tokens 124 -> 83 (34 % of the FMA rate), 4 x 4000 tokens 1016 -> 866.
#include <cooperative_groups.h>

#include "pbs_common.cuh"

namespace pbs {
namespace {

constexpr int FM = 32;        // query rows per CTA
constexpr int FN = 64;        // keys per step
constexpr int FT = 128;       // threads
constexpr int FP = FM + 4;    // floats per row of the P tile (key-major)

template <int D>
struct Fp32Smem {
  static constexpr int kLd = D + 4;                       // padded row: 16-byte reads of 8 neighbouring keys hit all banks
  static constexpr int kCtas = D == 64 ? 4 : 2;           // that a SM holds
  static constexpr int kFloats = FM * kLd + FN * (kLd + D) + FN * FP;
  static size_t bytes(int nb) { return sizeof(float) * kFloats + sizeof(int32_t) * FN + sizeof(uint16_t) * ((nb + 7) & ~7); }
};

__device__ __forceinline__ void cp16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}

template <int D>
__global__ void __launch_bounds__(FT, Fp32Smem<D>::kCtas)
attn_fp32_kernel(const float* __restrict__ q, Strides qs, const float* __restrict__ pk, const float* __restrict__ pv,
                 const int32_t* __restrict__ idx, const uint8_t* __restrict__ mask, float* __restrict__ out, Strides os,
                 int Hq, int S, int bs, int nb, int ranks, float scale_log2e) {
  using SM = Fp32Smem<D>;
  constexpr int LD = SM::kLd, C4 = D / 4, OC = D / 16;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                                         // [FM][LD]
  float* Ks = Qs + FM * LD;                               // [FN][LD]
  float* Vs = Ks + FN * LD;                               // [FN][D]
  float* Ps = Vs + FN * D;                                // [FN][FP]
  int32_t* kpos = reinterpret_cast<int32_t*>(Ps + FN * FP);               // [FN] original positions
  uint16_t* kept = reinterpret_cast<uint16_t*>(kpos + FN);                // kept blocks of this query block
  __shared__ int wcount[FT / 32];

  const int rank = blockIdx.x % ranks;                    // in the cluster of CTAs that shares the query tile's steps
  const int bh = blockIdx.x / ranks, b = bh / Hq, h = bh % Hq;
  const int r0 = (gridDim.y - 1 - blockIdx.y) * FM;       // the longest rows start first
  const int qb = r0 / bs;
  const float* qbase = q + (int64_t)b * qs.b + (int64_t)h * qs.h;
  const float* kbase = pk + (int64_t)bh * S * D;
  const float* vbase = pv + (int64_t)bh * S * D;
  const int32_t* ibase = idx + (int64_t)bh * S;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;

  for (int i = threadIdx.x; i < FM * C4; i += FT) {
    const int r = i / C4, c = i % C4;
    const bool live = r0 + r < S;
    cp16(Qs + r * LD + 4 * c, qbase + (int64_t)(live ? r0 + r : 0) * qs.s + 4 * c, live);
  }
  // the kept blocks, in order
  int nkept = 0;
  const uint8_t* mrow = mask + ((int64_t)bh * nb + qb) * nb;
  for (int k0 = 0; k0 < nb; k0 += FT) {
    const int kb = k0 + threadIdx.x;
    const bool on = kb < nb && mrow[kb];
    const unsigned ball = __ballot_sync(0xffffffffu, on);
    if (lane == 0) wcount[warp] = __popc(ball);
    __syncthreads();
    int at = nkept + __popc(ball & ((1u << lane) - 1));
    for (int w = 0; w < FT / 32; ++w) {
      if (w < warp) at += wcount[w];
      nkept += wcount[w];
    }
    if (on) kept[at] = (uint16_t)kb;
    __syncthreads();
  }
  // this CTA's steps: every ranks-th
  const int per_block = bs / FN, nsteps = (nkept * per_block - rank + ranks - 1) / ranks;
  auto first_key = [&](int s) {
    const int step = s * ranks + rank;
    return (int)kept[step / per_block] * bs + (step % per_block) * FN;
  };
  auto load = [&](int s) {
    const int k0 = first_key(s);
    for (int i = threadIdx.x; i < FN * C4; i += FT) {
      const int r = i / C4, c = i % C4;
      const bool live = k0 + r < S;
      const int64_t at = (int64_t)(live ? k0 + r : 0) * D + 4 * c;
      cp16(Ks + r * LD + 4 * c, kbase + at, live);
      cp16(Vs + r * D + 4 * c, vbase + at, live);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (threadIdx.x < FN) kpos[threadIdx.x] = k0 + (int)threadIdx.x < S ? ibase[k0 + threadIdx.x] : 0x7fffffff;
  };

  float2 acc[4][OC / 2];
  float m_run[4], l_run[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_run[i] = -CUDART_INF_F;
    l_run[i] = 0.f;
#pragma unroll
    for (int j = 0; j < OC / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
  }

  if (nsteps > 0) load(0);
  for (int s = 0; s < nsteps; ++s) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // S = Q K^T: rows 4 ty + i, keys tx + 16 j
    float2 sp[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sp[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 a[4], c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(Qs + (4 * ty + i) * LD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) c[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * LD + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sp[i][j] = __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(c[j].x, c[j].y), sp[i][j]);
          sp[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(c[j].z, c[j].w), sp[i][j]);
        }
    }
    // online softmax; every key's position counts, because the order of a stage call need not stay inside the segments
    int kp[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) kp[j] = kpos[tx + 16 * j];
    float p[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int qpos = r0 + 4 * ty + i;
      float mt = -CUDART_INF_F;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x = (sp[i][j].x + sp[i][j].y) * scale_log2e;
        if (kp[j] > qpos) x = -CUDART_INF_F;
        p[i][j] = x;
        mt = fmaxf(mt, x);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
      const float m_new = fmaxf(m_run[i], mt);
      const float m_ref = m_new == -CUDART_INF_F ? 0.f : m_new;      // nothing visible yet: every term is 0
      const float alpha = m_new == -CUDART_INF_F ? 1.f : exp2f(m_run[i] - m_new);
      float lt = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        p[i][j] = exp2f(p[i][j] - m_ref);
        lt += p[i][j];
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) lt += __shfl_xor_sync(0xffffffffu, lt, o);
      l_run[i] = l_run[i] * alpha + lt;
      m_run[i] = m_new;
#pragma unroll
      for (int j = 0; j < OC / 2; ++j) acc[i][j] = __fmul2_rn(acc[i][j], make_float2(alpha, alpha));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4*>(Ps + (tx + 16 * j) * FP + 4 * ty) = make_float4(p[0][j], p[1][j], p[2][j], p[3][j]);
    __syncwarp();                                         // the rows' 16 lanes are one half of a warp
    // O += P V: columns 4 tx (+ 64) .. + 3
#pragma unroll 4
    for (int kk = 0; kk < FN; ++kk) {
      const float4 pr = *reinterpret_cast<const float4*>(Ps + kk * FP + 4 * ty);
      const float pa[4] = {pr.x, pr.y, pr.z, pr.w};
#pragma unroll
      for (int jc = 0; jc < OC / 4; ++jc) {
        const float4 vv = *reinterpret_cast<const float4*>(Vs + kk * D + 64 * jc + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][2 * jc] = __ffma2_rn(make_float2(pa[i], pa[i]), make_float2(vv.x, vv.y), acc[i][2 * jc]);
          acc[i][2 * jc + 1] = __ffma2_rn(make_float2(pa[i], pa[i]), make_float2(vv.z, vv.w), acc[i][2 * jc + 1]);
        }
      }
    }
    __syncthreads();                                      // the tiles are free again
    if (s + 1 < nsteps) load(s + 1);
  }
  if (nsteps == 0) {                                      // the query tile's copies end before its place is used again
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
  float* obase = out + (int64_t)b * os.b + (int64_t)h * os.h;
  if (ranks == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = r0 + 4 * ty + i;
      if (row >= S) continue;
      const float inv = l_run[i] > 0.f ? 1.f / l_run[i] : 0.f;
#pragma unroll
      for (int jc = 0; jc < OC / 4; ++jc)
        *reinterpret_cast<float4*>(obase + (int64_t)row * os.s + 64 * jc + 4 * tx) =
            make_float4(acc[i][2 * jc].x * inv, acc[i][2 * jc].y * inv, acc[i][2 * jc + 1].x * inv, acc[i][2 * jc + 1].y * inv);
    }
    return;
  }
  // The CTAs' parts of O and their row statistics meet in shared memory (the Q tile's and the P tile's place); each CTA puts together and
  // stores every ranks-th row.
  float* part = Qs;                                       // [FM][LD]
  float2* stat = reinterpret_cast<float2*>(Ps);           // [FM] (maximum, sum)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int jc = 0; jc < OC / 4; ++jc)
      *reinterpret_cast<float4*>(part + (4 * ty + i) * LD + 64 * jc + 4 * tx) =
          make_float4(acc[i][2 * jc].x, acc[i][2 * jc].y, acc[i][2 * jc + 1].x, acc[i][2 * jc + 1].y);
    if (tx == 0) stat[4 * ty + i] = make_float2(m_run[i], l_run[i]);
  }
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int t = threadIdx.x; t < (FM / ranks) * C4; t += FT) {
    const int r = (t / C4) * ranks + rank, c = t % C4;
    if (r0 + r >= S) continue;
    float m = -CUDART_INF_F;
    for (int x = 0; x < ranks; ++x) m = fmaxf(m, cluster.map_shared_rank(stat, x)[r].x);
    const float m_ref = m == -CUDART_INF_F ? 0.f : m;
    float l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int x = 0; x < ranks; ++x) {
      const float2 st = cluster.map_shared_rank(stat, x)[r];
      const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, x) + r * LD + 4 * c);
      const float w = exp2f(st.x - m_ref);
      l += w * st.y;
      o.x += w * v.x; o.y += w * v.y; o.z += w * v.z; o.w += w * v.w;
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    *reinterpret_cast<float4*>(obase + (int64_t)(r0 + r) * os.s + 4 * c) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
  }
  cluster.sync();                                         // nobody leaves while its part is read
}

template <int D>
int run_fp32(const Dims& d, const void* q, Strides qs, const void* pk, const void* pv, const int32_t* idx, const uint8_t* mask,
             void* out, Strides os, cudaStream_t st) {
  const size_t smem = Fp32Smem<D>::bytes(d.nb);
  cudaError_t e = cudaFuncSetAttribute(attn_fp32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "attn_fp32_kernel smem attribute");
  // CTAs a query tile: as many as it takes to fill the GPU's places, at most 8 (a portable cluster) and one a step
  const int tiles = (d.S + FM - 1) / FM;
  int ranks = 1;
  while (ranks < 8 && ranks * FN < d.S && (int64_t)tiles * d.B * d.Hq * ranks < Fp32Smem<D>::kCtas * device_sms()) ranks *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(d.B * d.Hq * ranks, tiles);
  cfg.blockDim = dim3(FT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ranks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = ranks > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, attn_fp32_kernel<D>, (const float*)q, qs, (const float*)pk, (const float*)pv, idx, mask, (float*)out, os, d.Hq, d.S,
                         d.bs, d.nb, ranks, (float)(1.4426950408889634 / sqrt((double)d.D)));
  if (e != cudaSuccess) return cuda_fail(e, "attn_fp32_kernel");
  PBS_CUDA_CHECK_LAUNCH("attn_fp32_kernel");
  return PBS_OK;
}

}  // namespace

// Blocks must be whole steps.  The 4096 blocks a row that the library takes at most keep the row of kept blocks (8 KB) beside
// the CTAs' tiles and the query tiles within the grid's second dimension.
bool attn_fp32_supported(const Dims& d, int dt) {
  return dt == PBS_FP32 && (d.D == 64 || d.D == 128) && d.bs % FN == 0;
}

int launch_attn_fp32(const Dims& d, const void* q, Strides qs, const void* pk, const void* pv, const int32_t* idx,
                     const uint8_t* mask, void* out, Strides os, cudaStream_t st) {
  return d.D == 64 ? run_fp32<64>(d, q, qs, pk, pv, idx, mask, out, os, st)
                   : run_fp32<128>(d, q, qs, pk, pv, idx, mask, out, os, st);
}

}  // namespace pbs
