// Pooling of one block of query rows, for the kernel of its own and beside the first scoring pass.
#pragma once

#include "pbs_common.cuh"

namespace pbs {

// The rows of query block `blk` of one head (first row at qh, `row` elements apart) pooled into out[0 .. D), by `threads` threads that
// `sync` brings together.  A thread owns one 16-row group x one 16-byte piece of the row: LOADS of its loads are in flight at
// once, its sums follow the reference's reduction order (rows one after the other inside a group of 16); a second
// step adds the group sums in order.  part: [bs / 16][D] floats of shared memory.
template <int DT, int LOADS, typename Sync>
__device__ __forceinline__ void pool_query_block(const typename Elem<DT>::T* __restrict__ qh, int64_t row, typename Elem<DT>::T* __restrict__ out, int blk,
                                                 int pool_mode, int S, int D, int bs, float* part, int tid, int threads, Sync sync) {
  using E = Elem<DT>;
  using T = typename E::T;
  constexpr int EPV = 16 / (int)sizeof(T);
  const int r0 = blk * bs, r1 = min(r0 + bs, S);
  const int groups = bs / 16, cpr = D / EPV;
  const bool mean = pool_mode == PBS_POOL_MEAN;
  for (int i = tid; i < groups * cpr; i += threads) {
    const int g = i / cpr, c = i % cpr;
    const int g0 = r0 + 16 * g, n = max(0, min(16, r1 - g0));
    float acc[EPV];
#pragma unroll
    for (int t = 0; t < EPV; ++t) acc[t] = mean ? 0.f : -CUDART_INF_F;
#pragma unroll
    for (int rl = 0; rl < 16; rl += LOADS) {
      uint4 raw[LOADS];
#pragma unroll
      for (int rr = 0; rr < LOADS; ++rr)
        if (rl + rr < n) raw[rr] = *reinterpret_cast<const uint4*>(qh + (int64_t)(g0 + rl + rr) * row + c * EPV);
#pragma unroll
      for (int rr = 0; rr < LOADS; ++rr) {
        if (rl + rr < n) {
          const T* e = reinterpret_cast<const T*>(&raw[rr]);
#pragma unroll
          for (int t = 0; t < EPV; ++t) acc[t] = mean ? acc[t] + E::ld(e + t) : fmaxf(acc[t], E::ld(e + t));
        }
      }
    }
#pragma unroll
    for (int t = 0; t < EPV; ++t) part[g * D + c * EPV + t] = acc[t];
  }
  sync();
  for (int d = tid; d < D; d += threads) {
    float res;
    if (mean) {
      float a1 = 0.f;
      for (int g = 0; g < groups; ++g) a1 += part[g * D + d];
      res = a1 / (float)bs;
    } else {
      float m = (r1 - r0 < bs) ? 0.f : -CUDART_INF_F;     // zero padding takes part in the max
      for (int g = 0; g < groups; ++g) m = fmaxf(m, part[g * D + d]);
      res = m;
    }
    out[d] = E::cvt(res);
  }
}

// What the first scoring pass pools beside its own work; pooled: the kernels did.
struct QueryPooling {
  void* pooled_q;
  int mode;
  bool pooled;
};

}  // namespace pbs
