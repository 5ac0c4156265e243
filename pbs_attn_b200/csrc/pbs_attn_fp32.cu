// Stage 3b for fp32 inputs: block-sparse causal flash-attention forward on the CUDA cores, register-tiled.
//
// Same math as pbs_attn_simt.cu (pbs_attn/src/kernels/permuted_block_sparse_attention.py:7-90,241-311): fp32
// scores scaled by 1/sqrt(D), key visible iff its original position <= the query's, online softmax in base 2,
// fp32 accumulators.  There is no fp32 tensor-core path, so the bound is the fp32 FMA rate: 4*D FLOP per
// (query, key) of the kept blocks.  One CTA = 32 query rows; a step = 64 keys of one kept block, brought in by
// cp.async while the step before is computed (head_dim 64; at 128 two buffers would leave one CTA a SM).
// 128 threads as 8 x 16: a thread owns 4 rows x 4 keys of S and 4 rows x D/16 columns of O, so 32 packed FMA pairs feed
// on 8 shared-memory reads of 16 bytes, and the 16 lanes that share rows reduce them by shuffles and pass P through
// shared memory without a block-wide barrier.  The products of two neighbouring head-dim elements go into two partial
// sums (packed fp32 pairs), which are added at the end of the row.
// Measured against pbs_attn_simt.cu's kernel (one row and 8 keys a thread, operands re-read for every FMA), 2048 tokens, block 64:
// 4 heads of 64 (1.1 G FMA) 1079 -> 127 us, 8 heads of 128 (4.6 G FMA) 1955 -> 277 us = 33 TFLOP/s; 8192 tokens 8230 -> 1032
// and (block 128) 19880 -> 3456 us = 38 TFLOP/s.
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
  static constexpr int kBuf = D == 64 ? 2 : 1;
  static constexpr int kFloats = FM * kLd + kBuf * FN * (kLd + D) + FN * FP;
  static size_t bytes(int nb) { return sizeof(float) * kFloats + sizeof(int32_t) * kBuf * FN + sizeof(uint16_t) * ((nb + 7) & ~7); }
};

__device__ __forceinline__ void cp16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}

template <int D>
__global__ void __launch_bounds__(FT, 2)
attn_fp32_kernel(const float* __restrict__ q, Strides qs, const float* __restrict__ pk, const float* __restrict__ pv,
                 const int32_t* __restrict__ idx, const uint8_t* __restrict__ mask, float* __restrict__ out, Strides os,
                 int Hq, int S, int bs, int nb, float scale_log2e) {
  using SM = Fp32Smem<D>;
  constexpr int LD = SM::kLd, NBUF = SM::kBuf, C4 = D / 4, OC = D / 16;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                                         // [FM][LD]
  float* Ks = Qs + FM * LD;                               // [NBUF][FN][LD]
  float* Vs = Ks + NBUF * FN * LD;                        // [NBUF][FN][D]
  float* Ps = Vs + NBUF * FN * D;                         // [FN][FP]
  int32_t* kpos = reinterpret_cast<int32_t*>(Ps + FN * FP);               // [NBUF][FN] original positions
  uint16_t* kept = reinterpret_cast<uint16_t*>(kpos + NBUF * FN);         // kept blocks of this query block
  __shared__ int wcount[FT / 32];

  const int bh = blockIdx.x, b = bh / Hq, h = bh % Hq;
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
  const int per_block = bs / FN, nsteps = nkept * per_block;
  auto first_key = [&](int s) { return (int)kept[s / per_block] * bs + (s % per_block) * FN; };
  auto load = [&](int s) {
    const int k0 = first_key(s), buf = s % NBUF;
    for (int i = threadIdx.x; i < FN * C4; i += FT) {
      const int r = i / C4, c = i % C4;
      const bool live = k0 + r < S;
      const int64_t at = (int64_t)(live ? k0 + r : 0) * D + 4 * c;
      cp16(Ks + (buf * FN + r) * LD + 4 * c, kbase + at, live);
      cp16(Vs + (buf * FN + r) * D + 4 * c, vbase + at, live);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (threadIdx.x < FN) kpos[buf * FN + threadIdx.x] = k0 + (int)threadIdx.x < S ? ibase[k0 + threadIdx.x] : 0x7fffffff;
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
    if (NBUF == 2 && s + 1 < nsteps) {
      load(s + 1);                                        // into the buffer the step before last has left
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int buf = s % NBUF;
    const float* Kt = Ks + buf * FN * LD;
    const float* Vt = Vs + buf * FN * D;

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
      for (int j = 0; j < 4; ++j) c[j] = *reinterpret_cast<const float4*>(Kt + (tx + 16 * j) * LD + d);
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
    for (int j = 0; j < 4; ++j) kp[j] = kpos[buf * FN + tx + 16 * j];
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
        const float4 vv = *reinterpret_cast<const float4*>(Vt + kk * D + 64 * jc + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][2 * jc] = __ffma2_rn(make_float2(pa[i], pa[i]), make_float2(vv.x, vv.y), acc[i][2 * jc]);
          acc[i][2 * jc + 1] = __ffma2_rn(make_float2(pa[i], pa[i]), make_float2(vv.z, vv.w), acc[i][2 * jc + 1]);
        }
      }
    }
    __syncthreads();                                      // the buffer and the P tile are free again
    if (NBUF == 1 && s + 1 < nsteps) load(s + 1);
  }
  if (nsteps == 0) asm volatile("cp.async.wait_all;" ::: "memory");   // the query tile's copies end inside the CTA
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = r0 + 4 * ty + i;
    if (row >= S) continue;
    const float inv = l_run[i] > 0.f ? 1.f / l_run[i] : 0.f;
    float* orow = out + (int64_t)b * os.b + (int64_t)h * os.h + (int64_t)row * os.s;
#pragma unroll
    for (int jc = 0; jc < OC / 4; ++jc)
      *reinterpret_cast<float4*>(orow + 64 * jc + 4 * tx) =
          make_float4(acc[i][2 * jc].x * inv, acc[i][2 * jc].y * inv, acc[i][2 * jc + 1].x * inv, acc[i][2 * jc + 1].y * inv);
  }
}

template <int D>
int run_fp32(const Dims& d, const void* q, Strides qs, const void* pk, const void* pv, const int32_t* idx, const uint8_t* mask,
             void* out, Strides os, cudaStream_t st) {
  const size_t smem = Fp32Smem<D>::bytes(d.nb);
  cudaError_t e = cudaFuncSetAttribute(attn_fp32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "attn_fp32_kernel smem attribute");
  attn_fp32_kernel<D><<<dim3(d.B * d.Hq, (d.S + FM - 1) / FM), FT, smem, st>>>(
      (const float*)q, qs, (const float*)pk, (const float*)pv, idx, mask, (float*)out, os, d.Hq, d.S, d.bs, d.nb,
      (float)(1.4426950408889634 / sqrt((double)d.D)));
  PBS_CUDA_CHECK_LAUNCH("attn_fp32_kernel");
  return PBS_OK;
}

}  // namespace

// Blocks must be whole steps.  The 4096 blocks a row that the library takes at most keep the row of kept blocks (8 KB) beside
// two CTAs' tiles and the query tiles within the grid's second dimension.
bool attn_fp32_supported(const Dims& d, int dt) {
  return dt == PBS_FP32 && (d.D == 64 || d.D == 128) && d.bs % FN == 0;
}

int launch_attn_fp32(const Dims& d, const void* q, Strides qs, const void* pk, const void* pv, const int32_t* idx,
                     const uint8_t* mask, void* out, Strides os, cudaStream_t st) {
  return d.D == 64 ? run_fp32<64>(d, q, qs, pk, pv, idx, mask, out, os, st)
                   : run_fp32<128>(d, q, qs, pk, pv, idx, mask, out, os, st);
}

}  // namespace pbs
