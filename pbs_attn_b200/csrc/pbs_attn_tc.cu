// Stage 3b, Blackwell kernel: block-sparse causal flash-attention forward on tcgen05 tensor cores.
//
// Math follows the reference's Triton kernel (pbs_attn/src/kernels/permuted_block_sparse_attention.py
// :7-90,241-311): S = Q K^T accumulated in fp32, keys of the query tile's own segment are visible iff
// their original position <= the query's, online softmax in base 2, P rounded to the input dtype
// before P V, fp32 output accumulator, O / row-sum stored in the input dtype.
//
// Work item = 256 consecutive queries of one (b, h): two 128-row query tiles that share every K/V
// tile staged in shared memory.  The item's tile list (built by tile_list_kernel) names the 128-key
// tiles that either query tile selected.  A persistent CTA (one per SM) draws its items from a queue
// (in the stage call a CTA takes one entry of it) and walks them with twenty warps in four roles:
//   warp 0      draws the items and tells the other roles; TMA producer: Q tiles, then the list's tiles into a ring of two
//               stages, each with the V tile of an entry and the K tile of the next one (the issuers need these together)
//   warps 1, 3  MMA issuers, one per query tile.  A 128-key tile is two half-steps of 64 keys with
//               their own 64 TMEM columns: S_h = Q K_h^T (SS, both operands K-major, 128B swizzle,
//               M=128 N=64) and O += P_h V_h (TS: P_h read from TMEM, V MN-major from shared memory)
//   warp 2      owns the TMEM allocation (all 512 columns: per query tile S_0 S_1 (64 each) and O (128))
//   warps 4-19  softmax, a warpgroup per query tile and key half: per half-step tcgen05.ld S_h, exp2 relative to the row's
//               reference, row sum, P_h written back over the first 32 columns of S_h as packed 16-bit pairs.  The
//               first half's warpgroup also divides O by the row sum and stores it through a transposition tile
// K and V come through tensor maps of any strides with the query heads of a group on one head, so a call whose keys keep
// their order needs no copy of them (kernels of a call with and without, in turn: MeanPooling at 16384 tokens 1633 and 1564 us;
// 187 tokens 30.3 and 14.4, where one set-up kernel takes the place of gather, mask and list kernels).
// An issuer runs, per list entry and half h: O += P_h V_h, then S_h of the next entry into the
// columns P_h vacated.  One issuer's barrier bookkeeping overlaps the other issuer's MMAs.
//
// What bounds it.  At head_dim 128 TMEM has no room for a second S (at 64 it would have, unused), so each of the four (query tile, key half) chains S -> P -> P V -> next S
// is serial, and its latency is what counts: about 1300 cycles of softmax and as many of MMAs and hand-overs, while
// the tensor pipe needs 2560 cycles for the four (K = 16 of S at N = 64 takes 48 cycles and not 32, because shared memory
// delivers 128 bytes a cycle) and the special-function units 2048.  With one softmax warpgroup per query tile for both halves, as
// it was, a scheduler had two such warps, in step with each other more often than not, and the exponentials of one waited for the
// other's; with four there is nearly always one to run.  Measured (attention alone, in turn, 0.25 s blocks): 4 x 2048
// tokens 217 -> 198 us, 6001 sparse tokens fp16 243 -> 214, head_dim 64 382 -> 313, 8192 tokens 557 -> 527, block_size 64 at 32768
// tokens 7245 -> 6816, 32768 sparse tokens 4325 -> 3693, four heads at 131072 tokens 14255 -> 13800 (power cap).
// Three things make four warpgroups pay, each of which alone decides between a gain and a loss:
//  - the warps of the two halves exchange nothing from step to step.  A row's reference is not its running maximum
//    but what its first tile gave; it is raised only when a half-step's sum leaves kSumMost, which hardly
//    ever happens.  All of that protocol (settle, before_exp) is out of line.  With a check between the halves in every
//    half-step (a poll, an order of the hand-overs) the kernel was slower than before: 3200 to 3500 cycles a step against 2850.
//  - registers: 96 a thread at 640 threads, 104 after the issuing warps have given some up.  S is read in two parts of 32
//    columns; read at once it spills (2 % slower), in parts of 16 or with a part ahead it is slower too.
//  - nothing that does not need S stands between the wait for S and the arrive on P.
// Every wait on an mbarrier is bounded (2 s unless pbs_debug_set_attn_wait says otherwise); when one
// runs out the CTA raises a flag, all roles leave their loops, in-flight copies and MMAs are waited
// out (bounded), TMEM is freed and status[0] tells the host which wait it was.
#include <cuda.h>

#include <atomic>

#include "pbs_common.cuh"
#include "pbs_schedule.h"

namespace pbs {
namespace {

constexpr int kThreads = 640;
constexpr int kRing = 2;                  // stages of a V tile and the next list entry's K tile
constexpr int kSched = 4;                 // items the producer may be ahead of the slowest role
constexpr uint32_t kTmemCols = 512;
// A half-step's probabilities are taken as they are while their sum per row is no larger than this: the reference of the exponents need
// not be the row maximum, only near enough that nothing leaves its range.  For fp16 that is P's (65504).  For bf16 it is what V, which may be
// as large as fp32's numbers, leaves for O, the sum of P V before it is divided: with 2^8 |O| is at most 2^8 |V| a half-step.
// References that are raised often cost much (8192 tokens of head_dim 64 478 us a call, 577 with this limit and references at the
// maximum), so bf16's lie kLift above the maximum that they are taken from: scores may still rise by 2^20 (sum of 64), at
// which the rare path was as rare as with 2^60; at 2^14 32768 sparse tokens took 4579 us against 4385.  P and O of a row are
// then 2^-12 of what they could be, which leaves all of |V| down to fp32's least normal number its 8 bits in O.
template <int DT> constexpr float kSumMost = DT == PBS_FP16 ? 0x1p15f : 0x1p8f;
template <int DT> constexpr float kUpLeast = DT == PBS_FP16 ? 9.f : 2.f;    // log2(kSumMost / 64): a larger sum of 64 has a score above it
template <int DT> constexpr float kLift = DT == PBS_FP16 ? 0.f : 12.f;
// Registers a thread: the four warps that only issue give up part of what the launch has.
constexpr int kRegsLaunch = 96, kRegsIssue = 64, kRegsSoftmax = 104;
static_assert(128 * kRegsIssue + 512 * kRegsSoftmax <= kThreads * kRegsLaunch, "the shares must fit what the launch has");

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// One lane of a fully converged warp; the surrounding code stays warp-uniform, which lets the
// compiler keep descriptors and addresses in uniform registers.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .b32 rx;\n\t.reg .pred px;\n\t"
      "elect.sync rx|px, %1;\n\t"
      "@px mov.s32 %0, 1;\n\t}"
      : "+r"(pred)
      : "r"(0xFFFFFFFFu));
  return pred != 0;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// L2 eviction policies for the TMA loads: K/V tiles are re-read by every query group of the head
// (keep them), Q tiles are read once (let them go first).
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "l"(policy)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Executed by a converged warp; one elected lane commits.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  if (elect_one())
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], accumulate flag known at compile time (no predicate set-up).
template <bool ACC>
__device__ __forceinline__ void mma_ss_c(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  if (elect_one())
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0)
      : "memory");
}
template <bool ACC>
__device__ __forceinline__ void mma_ts_c(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
  if (elect_one())
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if (elect_one())
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1 (sm_100).
// lbo / sbo are byte offsets (multiples of 16).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two probabilities as the MMA takes them; `add` sums them up in fp32.  The row sum is that of the weights that P V uses, so that O / l is an
// average of V with weights that add up to one.  Relative error of a call against 64 bits, 1e-3, so / with the sum of the unrounded ones / with
// that and running maxima, as it was: 32768 sparse tokens 2.227 / 2.307 / 2.253, 8192 tokens of head_dim 64 2.184 / 2.254 / 2.256, 4 x 2048 2.064 /
// 2.096 / 2.133; lowest so in all 14 cases tried, fp16 among them.  (The unrounded sum takes 1 to 3 % less time.)
template <int DT> struct PackP;
template <> struct PackP<PBS_BF16> {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ void add(float2& a, uint32_t w) {
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.bf16 %0, lo, %0;\n\tadd.rn.f32.bf16 %1, hi, %1;\n\t}" : "+f"(a.x), "+f"(a.y) : "r"(w));
  }
  static __device__ __forceinline__ uint32_t scale(uint32_t w, float by) {
    const float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w));
    return pack(x.x * by, x.y * by);
  }
};
template <> struct PackP<PBS_FP16> {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ void add(float2& a, uint32_t w) {
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.f16 %0, lo, %0;\n\tadd.rn.f32.f16 %1, hi, %1;\n\t}" : "+f"(a.x), "+f"(a.y) : "r"(w));
  }
  static __device__ __forceinline__ uint32_t scale(uint32_t w, float by) {
    const float2 x = __half22float2(*reinterpret_cast<__half2*>(&w));
    return pack(x.x * by, x.y * by);
  }
};

// ---------------------------------------------------------------------------------------------
// Shared-memory plan
// ---------------------------------------------------------------------------------------------
struct Bars {
  uint64_t q_full[2], q_empty[2];
  uint64_t kv_full[kRing], kv_empty[kRing];
  uint64_t s_full[2][2], p_full[2][2], o_full[2][2];   // [query tile][key half]
  uint64_t l_full[2][4];                                // [query tile][lane quarter] row sums of the second key half are in lsum
  uint64_t start[2][4];                                 // [query tile][lane quarter] first maxima of both halves are in smax
  uint64_t item_full[kSched], item_empty[kSched];
  uint64_t drain;                                       // teardown after an abort: both issuers' MMAs retired
};

struct Params {
  const int32_t* idx;         // (B*Hq, S) original position of each key slot; null: the identity
  int kv_group;               // query heads that share a K/V head of the tensor maps
  const uint32_t* list;       // (B*Hq, G, T)
  const int32_t* count;       // (B*Hq, G)
  void* out;
  Strides os;
  int Hq, S, G, T;
  Schedule work;
  int bs;
  float scale_log2e;
  int32_t* status;
  int32_t* queue;               // draws so far, zero before and after a launch
  void* extra_out[PBS_MAX_OUT_REPLICAS];   // further destinations of the output (same strides), e.g. on peer GPUs
  int n_extra;
  unsigned long long wait_ns;   // limit of every device-side wait
  int drop_arrive;              // diagnostic: CTA 0's first softmax warpgroup (without a queue that of the first so many CTAs) skips one arrive
};

struct Ctl {
  int2 item[kSched];            // (b, h) and query group of the items handed to the other roles; x < 0: no more
  uint32_t tmem_base;
  volatile int abort_flag;
  // Shared by the two softmax warps (one per key half) of a query tile's lane quarter, see settle:
  uint2 post[2][2][4];          // [query tile][key half][lane quarter] progress, epoch of the references that its last P refers to
  uint32_t epoch[2][4];         // [query tile][lane quarter] times the references were raised
  uint32_t raised_at[2][2][4];  // [epoch & 1][query tile][lane quarter] half-step (2 * list entries done + key half) that raised them last
  float ref[2][2][128];         // [epoch & 1][query tile] references when they were raised last: the partner may still be reading the ones before
  float smax[2][2][2][128];     // [entry & 1][query tile][key half] first maxima
  uint32_t starts[2][2][4];     // [query tile][key half][lane quarter] meetings so far
  float lsum[2][128], lref[2][128];   // row sums of an item's second key half, and the references they are relative to
  unsigned long long wait_ns;
  int32_t* status;
};

template <int D>
struct Smem {
  static constexpr int kTileBytes = 128 * D * 2;          // one 128-row tile
  static constexpr int kQ = 0;                            // 2 tiles
  static constexpr int kV = kQ + 2 * kTileBytes;          // per stage a V tile and a K tile
  static constexpr int kK = kV + kTileBytes;
  static constexpr int kStage = 2 * kTileBytes;
  static constexpr int kEnd = kV + kRing * kStage;
};
constexpr int kStageRow = 80;                             // bytes per staged row piece (64 of data + 16 of padding)
// What does not depend on head_dim lies in front, at addresses known to the compiler.
struct __align__(1024) Front {
  Bars bars;
  Ctl ctl;
  alignas(16) int32_t kidx[16][64];                                   // key positions of a masked half tile, per softmax warp
  alignas(16) unsigned char stage[8][32 * kStageRow];                 // epilogue transposition, per lane quarter of a query tile
};
extern __shared__ __align__(1024) unsigned char smem_dyn[];
__device__ __forceinline__ Front& front() { return *reinterpret_cast<Front*>(smem_dyn); }
template <int D> constexpr int kSmemBytes = (int)sizeof(Front) + Smem<D>::kEnd;

// Bounded wait: false when the CTA is aborting (this wait or another one ran out of time).
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0u) {
      Ctl& ctl = front().ctl;
      if (ctl.abort_flag) return false;
      if (global_timer_ns() - t0 > ctl.wait_ns) {
        ctl.abort_flag = 1;
        atomicCAS(ctl.status, 0, code);
        return false;
      }
    }
  }
}

// The same for a whole converged warp: every lane polls, the verdict is made warp-uniform.
__device__ __forceinline__ bool wait_bar_warp(uint32_t bar, uint32_t parity, int code) {
  return __all_sync(0xffffffffu, wait_bar(bar, parity, code));
}

// Most waits pass at once: the rest is kept out of the hot loops' instruction stream.
__device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, int code) {
  return wait_bar_warp(bar, parity, code);
}
__device__ __forceinline__ bool wait_hot(uint32_t bar, uint32_t parity, int code) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return wait_slow(bar, parity, code);
}

// The 64 scores of this thread's row, in TMEM: those of keys after the query become -inf.
__device__ __noinline__ void mask_half(uint32_t s_addr, const int32_t* kidx, int qpos) {
#pragma unroll 1
  for (int c = 0; c < 64; c += 16) {
    uint32_t r[16];
    tmem_ld16(s_addr + c, r);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int4 k = *reinterpret_cast<const int4*>(kidx + c + 4 * j);
      if (k.x > qpos) r[4 * j] = 0xff800000u;
      if (k.y > qpos) r[4 * j + 1] = 0xff800000u;
      if (k.z > qpos) r[4 * j + 2] = 0xff800000u;
      if (k.w > qpos) r[4 * j + 3] = 0xff800000u;
    }
    tmem_st16(s_addr + c, r);
  }
  tmem_wait_st();
}

// This thread's row of O, in TMEM, times alpha.
__device__ __noinline__ void rescale_o(uint32_t o_addr, float alpha, int columns) {
#pragma unroll 1
  for (int c = 0; c < columns; c += 16) {
    uint32_t o[16];
    tmem_ld16(o_addr + c, o);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
    tmem_st16(o_addr + c, o);
  }
}

// P_h of this thread's row, in TMEM as packed pairs, times a power of two.
template <int DT>
__device__ __noinline__ void scale_p(uint32_t p_addr, float alpha) {
#pragma unroll 1
  for (int c = 0; c < 32; c += 16) {
    uint32_t r[16];
    tmem_ld16(p_addr + c, r);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = PackP<DT>::scale(r[j], alpha);
    tmem_st16(p_addr + c, r);
  }
}

// Waits (bounded) until a warp's progress is at least `least`.
__device__ __noinline__ bool wait_post(uint32_t addr, uint32_t least, uint2& post, int code) {
  Ctl& ctl = front().ctl;
  const uint64_t t0 = global_timer_ns();
  for (uint32_t it = 1;; ++it) {
    asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(post.x), "=r"(post.y) : "r"(addr) : "memory");
    if (__all_sync(0xffffffffu, post.x >= least)) return true;
    if ((it & 63u) == 0u && __any_sync(0xffffffffu, ctl.abort_flag || global_timer_ns() - t0 > ctl.wait_ns)) {
      ctl.abort_flag = 1;
      atomicCAS(ctl.status, 0, code);
      return false;
    }
  }
}

// Largest of the 64 scores of this thread's row, in TMEM.
__device__ __forceinline__ float row_max64(uint32_t s_addr) {
  float m = -CUDART_INF_F;
#pragma unroll
  for (int c = 0; c < 64; c += 32) {
    uint32_t r[32];
    tmem_ld32(s_addr + c, r);
    tmem_wait_ld();
    float a = m, b = m;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      a = max3(a, __uint_as_float(r[j]), __uint_as_float(r[j + 1]));
      b = max3(b, __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
    }
    m = fmaxf(a, b);
  }
  return m;
}

// The references of a softmax warp's rows.  Both warps of a lane quarter (one per key half) use the same; `ref` is log2 of the factor
// that the row's P, sum and O lack, -inf where the row has seen no key yet (then 0 is used, and everything is zero so far).
struct Refs {
  float ref, l;                                            // of this lane's row; l: row sum of this key half
  uint32_t epoch;                                          // times they were raised; kFresh: some row has none yet; kGiveUp: a wait ran out
};
constexpr uint32_t kFresh = 0x80000000u, kGiveUp = 0xffffffffu;
// A warp's progress (Ctl::post): 3 * list entries done, and more while it is in one of the functions below.
constexpr uint32_t kAtStart = 1, kRaising = 2;
__device__ __forceinline__ void st_post(uint32_t addr, uint32_t progress, uint32_t epoch) {
  asm volatile("st.volatile.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(progress), "r"(epoch) : "memory");
}

struct Who {                                               // of this softmax warp: query tile, key half, lane quarter; its lane's row
  int i, hs, wq, lane, row;
};
__device__ __forceinline__ Who who() {
  const int w = (int)(threadIdx.x >> 5) - 4, lane = threadIdx.x & 31;
  return Who{w >> 3, (w >> 2) & 1, w & 3, lane, (w & 3) * 32 + lane};
}

// 2^(from - to) for references of a row, `to` the later one: they are raised by whole numbers, so this is a power of two, or by more than
// 127, and then it is 0.
__device__ __forceinline__ float ref_scale(float from, float to) {
  const float n = rintf(from - to);
  return n >= -126.f ? __int_as_float(((int)fminf(n, 0.f) + 127) << 23) : 0.f;
}

// Takes over references that the partner warp has raised, up to epoch `now`.
__device__ __forceinline__ uint32_t epoch_of(const Who& w) { return *const_cast<const volatile uint32_t*>(&front().ctl.epoch[w.i][w.wq]); }
__device__ __forceinline__ void refresh(Refs& r, const Who& w, uint32_t now) {
  if (__any_sync(0xffffffffu, now != r.epoch)) {
    const float ref = *const_cast<const volatile float*>(&front().ctl.ref[now & 1u][w.i][w.row]);
    if (ref != r.ref && r.l > 0.f) r.l *= ref_scale(r.ref, ref);
    r.ref = ref;
    r.epoch = now;
  }
}

// Before the exponentials of a half-step whose keys are masked by position, or while some row has no reference: its first one is
// kLift above its largest score in both halves of the first tile that has one, so that the two warps meet here.
template <int DT>
__device__ __noinline__ Refs before_exp(Refs r, uint32_t ent, uint32_t tmem, uint32_t sc, bool none, bool first_entry, int qpos, float scale_log2e) {
  const Who w = who();
  Ctl& ctl = front().ctl;
  const uint32_t s_addr = tmem + ((uint32_t)(w.wq * 32) << 16) + 128 * w.i + 64 * w.hs;
  if (!none && (ent & (1u << (18 + w.i)))) mask_half(s_addr, front().kidx[(threadIdx.x >> 5) - 4], qpos);
  if (!(r.epoch & kFresh)) return r;
  // An item's first S was issued after all of the item before: nobody raises anything until both are past this meeting.  In a later entry
  // the first half may raise references in this very entry once it is past the meeting: what the second half takes over here is of before
  // that, so that its P is formed with the same references whether it is seen or not (settle); the first half needs all that the second has
  // raised in the entry before, which is complete when they meet.
  uint32_t epoch = epoch_of(w);
  r.epoch = first_entry ? epoch : r.epoch & ~kFresh;
  const float mine = none ? -CUDART_INF_F : row_max64(s_addr) * scale_log2e;
  if (w.lane == 0) st_post(smem_u32(&ctl.post[w.i][w.hs][w.wq]), 3u * sc + kAtStart, 0u);
  volatile float* both = &ctl.smax[sc & 1u][w.i][0][w.row];
  both[128 * w.hs] = mine;
  __threadfence_block();
  __syncwarp();
  const uint32_t bar = smem_u32(&front().bars.start[w.i][w.wq]);
  volatile uint32_t* starts = &ctl.starts[w.i][w.hs][w.wq];
  if (elect_one()) mbar_arrive(bar);
  if (!wait_bar_warp(bar, *starts & 1u, 14)) { r.epoch = kGiveUp; return r; }
  __syncwarp();
  if (w.lane == 0) *starts = *starts + 1u;
  __syncwarp();
  if (w.hs == 0) epoch = epoch_of(w);
  if (!first_entry) refresh(r, w, epoch);
  if (r.ref == -CUDART_INF_F) r.ref = fmaxf(mine, both[128 * (w.hs ^ 1)]) + kLift<DT>;
  if (__any_sync(0xffffffffu, r.ref == -CUDART_INF_F)) r.epoch |= kFresh;
  return r;
}

// References are raised by whole numbers, so that all is scaled by powers of two, exactly, and the result does not depend on who
// scales what and when.  Only where nothing is left of what was, by more than 127, to the maximum itself: from references of 10^10 (keys
// that a caller has pushed far down) a whole number leads to within a unit of 1024, not to the maximum.  A half-step k that finds a sum above
// kSumMost raises them: it waits for the P V of k - 1, which the old ones belong to, publishes the new ones and scales O.  S_k is still in TMEM, and since P_k has not been handed over, neither P V of k nor of the
// partner's k + 1 can start: O and P_{k+1} are its own.  P_{k+1} is always formed with the references before and then scaled.  Its warp reads
// the epoch after it has seen its S: if that S is not there yet it will see the new epoch and scale by itself.  Otherwise its
// progress says when it is through: with the old epoch its P is scaled here and its sum by itself once it sees the epoch; or it
// waits for the P V of k to raise references of its own, and takes the new ones after that.
// All of this is for half-steps that have seen another epoch or a sum above kSumMost; it forms and stores their P anew.
struct Settled {
  Refs r;
  float sum;
};
__device__ __forceinline__ bool raised_just_now(uint32_t now, const Who& w, uint32_t sc) {   // epoch `now` is the work of half-step k - 1
  return *const_cast<const volatile uint32_t*>(&front().ctl.raised_at[now & 1u][w.i][w.wq]) + 1u == 2u * sc + w.hs;
}
template <int DT, int D>
__device__ __noinline__ Settled settle(Refs r, uint32_t tmem, uint32_t sc, bool first_entry, float scale_log2e) {
  const Who w = who();
  Bars& bars = front().bars;
  Ctl& ctl = front().ctl;
  const uint32_t fresh = r.epoch & kFresh;
  r.epoch &= ~kFresh;
  const uint32_t lanes = (uint32_t)(w.wq * 32) << 16, s_addr = tmem + lanes + 128 * w.i + 64 * w.hs;
  auto given_up = [&]() {
    r.epoch = kGiveUp;
    return Settled{r, 0.f};
  };
  // P_k with the references in r, as the hot loop forms it; what is stored is scaled by alpha, the sum of the row is not.  Storing goes behind
  // reading: 16 scores give 8 columns of P.
  auto form = [&](bool store, float alpha) {
    const float ref = r.ref == -CUDART_INF_F ? 0.f : r.ref;
    const float2 sc2 = make_float2(scale_log2e, scale_log2e), nm2 = make_float2(-ref, -ref);
    float2 acc2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      uint32_t sr[16], pk[8];
      tmem_ld16(s_addr + 16 * q, sr);
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float2 x = __ffma2_rn(make_float2(__uint_as_float(sr[2 * c]), __uint_as_float(sr[2 * c + 1])), sc2, nm2);
        pk[c] = PackP<DT>::pack(ex2(x.x), ex2(x.y));
        PackP<DT>::add(acc2[c & 1], pk[c]);
        if (alpha != 1.f) pk[c] = PackP<DT>::scale(pk[c], alpha);
      }
      if (store) tmem_st8(s_addr + 8 * q, pk);
    }
    return (acc2[0].x + acc2[0].y) + (acc2[1].x + acc2[1].y);
  };
  auto refs_of = [&](uint32_t epoch) { return *const_cast<const volatile float*>(&ctl.ref[epoch & 1u][w.i][w.row]); };
  auto take = [&](uint32_t epoch) {
    const float ref = refs_of(epoch);
    if (ref != r.ref && r.l > 0.f) r.l *= ref_scale(r.ref, ref);
    r.ref = ref;
    r.epoch = epoch;
  };
  bool late = false;                                       // half-step k - 1 raised the references; P_k is formed with the ones before
  for (;;) {
    const uint32_t now = epoch_of(w);
    if (!__any_sync(0xffffffffu, now != r.epoch)) break;
    late = raised_just_now(now, w, sc);
    if (late && now == r.epoch + 1u) break;
    take(late ? now - 1u : now);
  }
  float sum = form(false, 1.f);
  if (!__any_sync(0xffffffffu, !(sum <= kSumMost<DT>))) {
    float alpha = 1.f;
    const Refs formed = r;
    if (late) {
      refresh(r, w, epoch_of(w));
      if (r.ref != formed.ref) alpha = ref_scale(formed.ref, r.ref);
    }
    const Refs after_it = r;
    r = formed;
    sum = form(true, alpha) * alpha;
    r = after_it;
    r.epoch |= fresh;
    return Settled{r, sum};
  }
  const uint32_t before = w.hs == 0 ? sc - 1u : sc, after = w.hs == 0 ? sc : sc + 1u;   // entries of half-steps k - 1 and k + 1
  const float top = row_max64(s_addr) * scale_log2e;
  if (w.lane == 0) st_post(smem_u32(&ctl.post[w.i][w.hs][w.wq]), 3u * sc + kRaising, r.epoch);
  const bool have_o = !first_entry || w.hs == 1;
  if (have_o) {
    if (!wait_bar_warp(smem_u32(&bars.o_full[w.i][w.hs ^ 1]), before & 1u, 10)) return given_up();
    tc_fence_after();
    refresh(r, w, epoch_of(w));
  }
  const bool up = top > r.ref + kUpLeast<DT>;
  if (__any_sync(0xffffffffu, up)) {
    const float old = r.ref;
    if (up) r.ref = (top - r.ref > 127.f ? top : r.ref + ceilf(top - r.ref)) + kLift<DT>;
    const float alpha = up ? ref_scale(old, r.ref) : 1.f;
    r.l *= alpha;
    ++r.epoch;
    *const_cast<volatile float*>(&ctl.ref[r.epoch & 1u][w.i][w.row]) = r.ref;
    if (w.lane == 0) *const_cast<volatile uint32_t*>(&ctl.raised_at[r.epoch & 1u][w.i][w.wq]) = 2u * sc + w.hs;
    __threadfence_block();
    __syncwarp();
    if (w.lane == 0) *const_cast<volatile uint32_t*>(&ctl.epoch[w.i][w.wq]) = r.epoch;
    __threadfence_block();
    __syncwarp();
    if (have_o) rescale_o(tmem + lanes + 256 + 128 * w.i, alpha, D);
    if (__all_sync(0xffffffffu, mbar_try_wait(smem_u32(&bars.s_full[w.i][w.hs ^ 1]), after & 1u))) {
      // (a first half has met the second one of its entry already)
      uint2 theirs;
      if (!wait_post(smem_u32(&ctl.post[w.i][w.hs ^ 1][w.wq]), 3u * after + (w.hs == 0 ? kRaising : kAtStart), theirs, 16)) return given_up();
      if (theirs.x >= 3u * (after + 1u) && theirs.y != r.epoch) {
        tc_fence_after();
        scale_p<DT>(tmem + lanes + 128 * w.i + 64 * (w.hs ^ 1), alpha);
      }
    }
  }
  sum = form(true, 1.f);
  r.epoch |= fresh;
  return Settled{r, sum};
}

// The n-th item of this CTA, for the roles that the producer feeds (a whole converged warp calls it).
// False past the last one, or when a wait ran out (then ok is false).
__device__ __forceinline__ bool next_item(int n, bool& ok, int& bh, int& g) {
  const int s = n % kSched;
  Bars* bars = &front().bars;
  Ctl* ctl = &front().ctl;
  ok = wait_bar_warp(smem_u32(&bars->item_full[s]), (n / kSched) & 1u, 12);
  if (!ok) return false;
  const int2 it = ctl->item[s];
  __syncwarp();
  if (elect_one()) mbar_arrive(smem_u32(&bars->item_empty[s]));
  bh = it.x;
  g = it.y;
  return bh >= 0;
}

// ---------------------------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------------------------
// QUEUE: CTAs draw their work with the counter p.queue; else each has one entry.  Its own instance, because the test in the
// kernel cost the whole-path call 0.1 to 0.5 %.
template <int DT, int D, bool QUEUE>
__global__ void __launch_bounds__(kThreads, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, Params p) {
  using E = Elem<DT>;
  using T = typename E::T;
  using SM = Smem<D>;
  const uint32_t sbase = smem_u32(smem_dyn) + (uint32_t)sizeof(Front);
  Bars* bars = &front().bars;
  Ctl* ctl = &front().ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars->q_full[i]), 1);
      mbar_init(smem_u32(&bars->q_empty[i]), 1);
      for (int h = 0; h < 2; ++h) {
        mbar_init(smem_u32(&bars->s_full[i][h]), 1);
        mbar_init(smem_u32(&bars->p_full[i][h]), 128);
        mbar_init(smem_u32(&bars->o_full[i][h]), 1);
      }
    }
    for (int i = 0; i < kRing; ++i) { mbar_init(smem_u32(&bars->kv_full[i]), 1); mbar_init(smem_u32(&bars->kv_empty[i]), 2); }
    for (int i = 0; i < kSched; ++i) { mbar_init(smem_u32(&bars->item_full[i]), 1); mbar_init(smem_u32(&bars->item_empty[i]), 18); }
    for (int i = 0; i < 2; ++i)
      for (int wq = 0; wq < 4; ++wq) {
        mbar_init(smem_u32(&bars->l_full[i][wq]), 1);
        mbar_init(smem_u32(&bars->start[i][wq]), 2);
        ctl->epoch[i][wq] = 0u;
        for (int h = 0; h < 2; ++h) { ctl->post[i][h][wq] = make_uint2(0u, 0u); ctl->starts[i][h][wq] = 0u; }
      }
    mbar_init(smem_u32(&bars->drain), 2);
    // Without a queue a CTA that starts after another one gave up need not wait out the limit as well (the result is invalid
    // already): its waits give up at once, so that a launch of many CTAs ends soon after the first of them.
    ctl->abort_flag = !QUEUE && blockIdx.x >= 1 && *const_cast<const volatile int32_t*>(p.status) != 0;
    ctl->wait_ns = p.wait_ns;
    ctl->status = p.status;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  const uint32_t tmem_S[2] = {tmem + 0u, tmem + 128u};
  const uint32_t tmem_O[2] = {tmem + 256u, tmem + 384u};

  constexpr int KH = D / 64;                              // 64-column (128-byte) slabs per tile row
  constexpr uint32_t kSlab = 128 * 128;                   // bytes of one 128-row slab
  constexpr uint32_t kTile = SM::kTileBytes;
  // instruction descriptors: fp32 accumulate, A/B = bf16 or fp16, M = 128
  constexpr uint32_t kFmt = (DT == PBS_BF16) ? 1u : 0u;
  constexpr uint32_t kIdescQK = (1u << 4) | (kFmt << 7) | (kFmt << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);   // N = 64
  constexpr uint32_t kIdescPV = (1u << 4) | (kFmt << 7) | (kFmt << 10) | (1u << 16) | (((uint32_t)D >> 3) << 17) | ((128u >> 4) << 24);


  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
  if (warp == 0) {
    // =========================================================================== TMA producer
    // The whole warp walks the lists (uniform control flow); one elected lane issues the copies.
    {
      uint32_t rc = 0, qc[2] = {0, 0};
      bool ok = true;
      const uint64_t pol_kv = l2_policy_evict_last(), pol_q = l2_policy_evict_first();
      // The items of this CTA: its first queue entry is its own number, each further one (of a queue) is drawn while
      // the entry before it is loaded.
      int q = (int)blockIdx.x, q_next = 0, j = 0;
      for (int it = 0, bh, g; ok; ++it) {
        const bool more = queue_item(p.work, q, j, bh, g);
        if (more && j == 0 && elect_one()) {
          if constexpr (QUEUE) {
            // one draw per entry of the queue; the last one leaves the counter at zero
            const int drawn = atomicAdd(p.queue, 1);
            if (drawn == entries(p.work) - 1) atomicExch(p.queue, 0);
            q_next = (int)gridDim.x + drawn;
          } else {
            q_next = p.work.n_items;                       // past the end
          }
        }
        ok = wait_bar_warp(smem_u32(&bars->item_empty[it % kSched]), ((it / kSched) & 1u) ^ 1u, 13);
        if (!ok) break;
        if (elect_one()) {
          ctl->item[it % kSched] = more ? make_int2(bh, g) : make_int2(-1, 0);
          mbar_arrive(smem_u32(&bars->item_full[it % kSched]));
        }
        if (!more) break;
        const int b = bh / p.Hq, h = bh % p.Hq;
        for (int i = 0; i < 2 && ok; ++i) {
          const int r0 = g * 256 + i * 128;
          if (r0 >= p.S) continue;
          ok = wait_bar_warp(smem_u32(&bars->q_empty[i]), (qc[i] & 1u) ^ 1u, 1);
          if (!ok) break;
          const uint32_t bar = smem_u32(&bars->q_full[i]);
          if (elect_one()) {
            mbar_expect_tx(bar, kTile);
            for (int kh = 0; kh < KH; ++kh)
              tma_load_4d(sbase + SM::kQ + i * kTile + kh * kSlab, &map_q, bar, kh * 64, r0, h, b, pol_q);
          }
          ++qc[i];
        }
        const int n = p.count[(int64_t)bh * p.G + g];
        const uint32_t* lst = p.list + ((int64_t)bh * p.G + g) * p.T;
        uint32_t ent = 0u, nxt = n > 0 ? lst[0] : 0u;
        for (int e = -1; e < n && n > 0 && ok; ++e) {      // V of entry e and K of entry e + 1
          const uint32_t nn = e + 2 < n ? lst[e + 2] : 0u; // read one entry ahead of its use
          const uint32_t s = rc % kRing;
          ok = wait_bar_warp(smem_u32(&bars->kv_empty[s]), ((rc / kRing) & 1u) ^ 1u, 2);
          if (!ok) break;
          const uint32_t bar = smem_u32(&bars->kv_full[s]);
          const bool have_v = e >= 0, have_k = e + 1 < n;
          if (elect_one()) {
            mbar_expect_tx(bar, (have_v && have_k ? 2 : 1) * kTile);
            if (have_v)
              for (int kh = 0; kh < KH; ++kh)
                tma_load_4d(sbase + SM::kV + s * SM::kStage + kh * kSlab, &map_v, bar, kh * 64, (int)(ent & 0xFFFFu) * 128, h / p.kv_group, b, pol_kv);
            if (have_k)
              for (int kh = 0; kh < KH; ++kh)
                tma_load_4d(sbase + SM::kK + s * SM::kStage + kh * kSlab, &map_k, bar, kh * 64, (int)(nxt & 0xFFFFu) * 128, h / p.kv_group, b, pol_kv);
          }
          ++rc;
          ent = nxt;
          nxt = nn;
        }
        if (j == 0 && q < p.work.pairs) {
          j = 1;
        } else {
          j = 0;
          q = __reduce_max_sync(0xffffffffu, q_next);      // only the elected lane has drawn, the others hold 0
          q_next = 0;
        }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // =========================================================================== MMA issuers
    // Warp 1 issues for query tile 0, warp 3 for query tile 1.  Control flow is uniform for the
    // whole warp; each tcgen05.mma / commit is issued by one elected lane.  Both warps walk the
    // whole list (the K/V ring is indexed by list position) and act on the entries their tile uses;
    // a ring stage is free again once BOTH have committed on its `empty` barrier.  The bookkeeping
    // of one warp (barrier waits, list reads) overlaps the other warp's MMAs on the tensor pipe.
    {
      const int i = warp >> 1;                              // query tile of this issuer
      uint32_t rc = 0, qc = 0, pc = 0;
      bool ok = true;
      const uint32_t use_bit = 1u << (16 + i);

      // Descriptors are built once; per instruction only a compile-time constant is added to the
      // start-address field.
      const uint64_t dq = smem_desc(sbase + SM::kQ + i * kTile, 16, 1024);
      const uint32_t bar_sfull[2] = {smem_u32(&bars->s_full[i][0]), smem_u32(&bars->s_full[i][1])};
      const uint32_t bar_ofull[2] = {smem_u32(&bars->o_full[i][0]), smem_u32(&bars->o_full[i][1])};
      const uint32_t tS = tmem_S[i], tO = tmem_O[i];

      // A 128-key tile is processed as two half-steps of 64 keys (h = 0, 1), each with its own 64
      // columns of S, so that the softmax of one half overlaps the MMAs of the other.
      // S_h = Q K_h^T: M = 128, N = 64; K_h = rows 64h .. 64h+63 of the staged K tile.
      auto issue_qk = [&](uint32_t kstage, int h) {
        const uint64_t b0 = smem_desc(sbase + SM::kK + kstage * SM::kStage + h * 64 * 128, 16, 1024);
        const uint32_t d = tS + 64 * h;
        mma_ss_c<false>(d, dq, b0, kIdescQK);
#pragma unroll
        for (int ks = 1; ks < D / 16; ++ks) {
          const uint64_t off = (uint64_t)(((ks >> 2) * kSlab + (ks & 3) * 32) >> 4);
          mma_ss_c<true>(d, dq + off, b0 + off, kIdescQK);
        }
        tc_commit(bar_sfull[h]);
      };
      // O += P_h V_h: P_h (64 keys as 32 columns of 16-bit pairs) sits in the first half of S_h.
      auto issue_pv = [&](uint32_t vstage, bool accumulate, int h) {
        const uint64_t b0 = smem_desc(sbase + SM::kV + vstage * SM::kStage, kSlab, 1024) + (uint64_t)h * ((4 * 2048) >> 4);
        const uint32_t a0 = tS + 64 * h;
        mma_ts(tO, a0, b0, kIdescPV, accumulate);
#pragma unroll
        for (int ks = 1; ks < 4; ++ks) mma_ts_c<true>(tO, a0 + ks * 8, b0 + (uint64_t)((ks * 2048) >> 4), kIdescPV);
        tc_commit(bar_ofull[h]);
      };

      for (int it = 0, bh, g; ok && next_item(it, ok, bh, g); ++it) {
        const int n = p.count[(int64_t)bh * p.G + g];
        const uint32_t* lst = p.list + ((int64_t)bh * p.G + g) * p.T;
        const bool have = g * 256 + i * 128 < p.S;
        if (have) {
          ok = wait_bar_warp(smem_u32(&bars->q_full[i]), qc & 1u, 4);
          ++qc;
          if (!ok) break;
        }
        bool started = false;                               // O_i holds a partial sum of this item
        uint32_t cur = 0u, nxt = n > 0 ? lst[0] : 0u;
        for (int e = -1; e < n && n > 0 && ok; ++e) {
          const uint32_t nn = (e + 2 < n) ? lst[e + 2] : 0u;    // read one entry ahead of its use
          // A stage's `full` barrier is awaited even when this tile skips both entries: an issuer must
          // not arrive on `empty` for a later round of the stage before the other issuer has arrived
          // for this one.
          const uint32_t s = rc % kRing;
          ok = wait_bar_warp(smem_u32(&bars->kv_full[s]), (rc / kRing) & 1u, 5);
          if (!ok) break;
          // per half: O += P_h V_h of this entry, then S_h of the next entry into the columns that
          // P_h just vacated
#pragma unroll
          for (int h = 0; h < 2 && ok; ++h) {
            if (cur & use_bit) {
              ok = wait_bar_warp(smem_u32(&bars->p_full[i][h]), pc & 1u, 7);
              if (!ok) break;
            }
            tc_fence_after();
            if (cur & use_bit) issue_pv(s, started || h == 1, h);
            if (nxt & use_bit) issue_qk(s, h);
          }
          if (!ok) break;
          if (cur & use_bit) {
            ++pc;
            started = true;
          }
          tc_commit(smem_u32(&bars->kv_empty[s]));
          ++rc;
          cur = nxt;
          nxt = nn;
        }
        if (!ok) break;
        if (have) tc_commit(smem_u32(&bars->q_empty[i]));
      }
      // Abort path: this commit arrives once every MMA this warp issued has retired.
      if (ctl->abort_flag) tc_commit(smem_u32(&bars->drain));
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    // =========================================================================== softmax + epilogue
    const int i = (warp - 4) >> 3;                         // query tile of this warpgroup
    const int hs = ((warp - 4) >> 2) & 1;                  // key half of this warpgroup
    const int wq = warp & 3;                               // TMEM lane quarter of this warp
    const int row = wq * 32 + lane;
    const uint32_t lane_off = (uint32_t)(wq * 32) << 16;
    const uint32_t s_addr = tmem + 128 * i + lane_off + 64 * hs;
    const uint32_t bar_s = smem_u32(&bars->s_full[i][hs]), bar_p = smem_u32(&bars->p_full[i][hs]);
    const uint32_t post = smem_u32(&ctl->post[i][hs][wq]);
    uint32_t sc = 0, sums = 0;                             // list entries done, row sums handed over
    bool ok = true;

    for (int it = 0, bh, g; ok && next_item(it, ok, bh, g); ++it) {
      const int r0 = g * 256 + i * 128;
      if (r0 >= p.S) continue;
      const uint32_t* lst = p.list + ((int64_t)bh * p.G + g) * p.T;
      const uint32_t* end = lst + p.count[(int64_t)bh * p.G + g];
      Refs r{-CUDART_INF_F, 0.f, kFresh};
      const uint32_t sc0 = sc;

      uint32_t ent_next = lst < end ? *lst : 0u;
      while (lst < end) {
        const uint32_t ent = ent_next;
        if (++lst < end) ent_next = *lst;                  // fetched one entry ahead of its use
        if (!(ent & (1u << (16 + i)))) continue;
        // with block_size 64 these rows may not attend this key half at all
        const bool none = p.bs == 64 && !((ent >> (20 + 4 * i + 2 * (wq >> 1) + hs)) & 1u);
        if (ent & (1u << (18 + i))) {                      // to be masked by position
          const int32_t* ibase = p.idx ? p.idx + (int64_t)bh * p.S : nullptr;
          int32_t* kidx = front().kidx[warp - 4];
          const int k0 = (int)(ent & 0xFFFFu) * 128 + 64 * hs + lane;
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 64; c += 32) kidx[c + lane] = k0 + c >= p.S ? 0x7fffffff : ibase ? ibase[k0 + c] : k0 + c;
          __syncwarp();
        }
        const bool cold = (ent & (1u << (18 + i))) || (r.epoch & kFresh);
        // diagnostic hook of the failure-path tests: the very first hand-over of a CTA is withheld, so the issuer's wait
        // for it runs out and the CTA takes the abort path
        const bool drop = p.drop_arrive && (QUEUE ? blockIdx.x == 0 : (int)blockIdx.x < p.drop_arrive) && sc == 0 && i == 0 && hs == 0;
        ok = wait_hot(bar_s, sc & 1u, 9);
        if (!ok) break;
        tc_fence_after();
        if (cold) {
          r = before_exp<DT>(r, ent, tmem, sc, none, sc == sc0, r0 + row, p.scale_log2e);
          ok = r.epoch != kGiveUp;
          if (!ok) break;
        }
        float sum = 0.f;
        if (none) {
          uint32_t zero[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) zero[c] = 0u;
          tmem_st32(s_addr, zero);
        } else {
          // All of P_h is formed before any of it goes back over the first 32 columns of S_h, so that S_h is still there when
          // the references turn out to be stale or too low.
          uint32_t pk[32], epoch_now;
          const float2 sc2 = make_float2(p.scale_log2e, p.scale_log2e);
          const float ref = r.ref == -CUDART_INF_F ? 0.f : r.ref;
          const float2 nm2 = make_float2(-ref, -ref);
          float2 acc2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t sr[32];
            tmem_ld32(s_addr + 32 * q, sr);
            // (the epoch is read after S is there: see settle)
            if (q == 0) asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(epoch_now) : "r"(smem_u32(&ctl->epoch[i][wq])) : "memory");
            tmem_wait_ld();
            float (&v)[32] = *reinterpret_cast<float (*)[32]>(&sr[0]);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const float2 x = __ffma2_rn(make_float2(v[2 * c], v[2 * c + 1]), sc2, nm2);
              const float2 ex = make_float2(ex2(x.x), ex2(x.y));
              pk[16 * q + c] = PackP<DT>::pack(ex.x, ex.y);
              PackP<DT>::add(acc2[c & 1], pk[16 * q + c]);
            }
          }
          sum = (acc2[0].x + acc2[0].y) + (acc2[1].x + acc2[1].y);
          if (!__any_sync(0xffffffffu, epoch_now != (r.epoch & ~kFresh) || !(sum <= kSumMost<DT>))) {
            tmem_st32(s_addr, pk);
          } else {
            const Settled settled = settle<DT, D>(r, tmem, sc, sc == sc0, p.scale_log2e);
            r = settled.r;
            sum = settled.sum;
            ok = r.epoch != kGiveUp;
            if (!ok) break;
          }
        }
        tmem_wait_st();
        tc_fence_before();
        if (!drop) mbar_arrive(bar_p);
        ++sc;
        if (lane == 0) st_post(post, 3u * sc, r.epoch & ~kFresh);
        r.l += sum;
      }
      if (!ok) break;
      const bool steps = sc != sc0;

      // The second half's warps hand their row sums to the first half's, which write the result.
      if (hs == 1) {
        if (steps) {
          *(volatile float*)&ctl->lsum[i][row] = r.l;
          *(volatile float*)&ctl->lref[i][row] = r.ref;
          __threadfence_block();
          __syncwarp();
          if (elect_one()) mbar_arrive(smem_u32(&bars->l_full[i][wq]));
        }
        continue;
      }
      if (steps) {
        ok = wait_hot(smem_u32(&bars->l_full[i][wq]), sums & 1u, 15);
        if (!ok) break;
        ++sums;
        // either half may have raised the references after the other's last step
        r.epoch &= ~kFresh;
        refresh(r, who(), epoch_of(who()));
        const float l1 = *(volatile float*)&ctl->lsum[i][row], ref1 = *(volatile float*)&ctl->lref[i][row];
        r.l += ref1 == r.ref || l1 == 0.f ? l1 : l1 * ref_scale(ref1, r.ref);
      }
      const int b = bh / p.Hq, h = bh % p.Hq;
      const uint32_t bar_o1 = smem_u32(&bars->o_full[i][1]);

      // epilogue: O / l in the input dtype, original token order (queries are not permuted)
      if (steps) {
        ok = wait_hot(bar_o1, (sc - 1u) & 1u, 11);
        if (!ok) break;
        tc_fence_after();
      }
      // Rows leave through a per-warp transposition tile: a thread owns one row of O in TMEM, but four
      // lanes then store one row's 64-byte piece together, so a store instruction writes 8 rows x 64
      // contiguous bytes instead of 32 rows x 16 -- this matters for the replicas, which travel over NVLink.
      const float inv = r.l > 0.f ? 1.f / r.l : 0.f;
      unsigned char* stage = front().stage[i * 4 + wq];
      const int64_t obase = (int64_t)b * p.os.b + (int64_t)h * p.os.h;
      const int wrow0 = r0 + wq * 32;                      // first query row of this warp
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t o[32];
        if (steps) {
          tmem_ld32(tmem_O[i] + lane_off + c * 32, o);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 w;
          w.x = PackP<DT>::pack(__uint_as_float(o[8 * j + 0]) * inv, __uint_as_float(o[8 * j + 1]) * inv);
          w.y = PackP<DT>::pack(__uint_as_float(o[8 * j + 2]) * inv, __uint_as_float(o[8 * j + 3]) * inv);
          w.z = PackP<DT>::pack(__uint_as_float(o[8 * j + 4]) * inv, __uint_as_float(o[8 * j + 5]) * inv);
          w.w = PackP<DT>::pack(__uint_as_float(o[8 * j + 6]) * inv, __uint_as_float(o[8 * j + 7]) * inv);
          *reinterpret_cast<uint4*>(stage + lane * kStageRow + j * 16) = w;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int rr = (lane >> 2) + 8 * j, piece = lane & 3;
          const int grow = wrow0 + rr;
          if (grow < p.S) {
            const uint4 w = *reinterpret_cast<const uint4*>(stage + rr * kStageRow + piece * 16);
            const int64_t off = obase + (int64_t)grow * p.os.s + c * 32 + piece * 8;
            __stcs(reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + off), w);   // written once, not re-read here
            // replicas (peer GPUs of a head-sharded call): plain stores, they travel over NVLink
            for (int x = 0; x < p.n_extra; ++x)
              *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.extra_out[x]) + off) = w;
          }
        }
        __syncwarp();
      }
      // the next item's first P V overwrites O_i: order our TMEM reads before the arrive that lets it go
      tc_fence_before();
    }
  }

  // =============================================================================== teardown
  // After an abort, work may still be in flight when the roles leave their loops: TMA copies into
  // this CTA's shared memory and MMAs into its TMEM.  Neither may outlive the CTA, so everybody
  // first lets the copies land (a copy takes a few microseconds; 100 us, bounded) and the TMEM owner
  // waits (bounded again) until both issuers' MMAs have retired before it frees the columns.
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (ctl->abort_flag) {
    for (int n = 0; n < 100; ++n) __nanosleep(1000);
    if (warp == 2) {
      const uint64_t t0 = global_timer_ns();
      while (!mbar_try_wait(smem_u32(&bars->drain), 0) && global_timer_ns() - t0 < 2000000ull) { }
      tc_fence_after();
    }
    __syncthreads();
  }
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
// Limit of every device-side wait and the diagnostic hook, process wide (pbs_debug_set_attn_wait).
std::atomic<unsigned long long> g_wait_ns{2000000000ull};
std::atomic<int> g_drop_arrive{0};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// Tensor map of a (B, heads, S, D) operand with 128-row boxes; the strides of size-1 dimensions are made up.
int make_map(CUtensorMap* map, int dt, const void* base, const Dims& d, int heads, Strides st) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) { set_error("cuTensorMapEncodeTiled is not available from the driver"); return PBS_ERR_CUDA; }
  const cuuint64_t row = (cuuint64_t)st.s * 2;
  const cuuint64_t sh = heads > 1 ? (cuuint64_t)st.h * 2 : row * d.S;
  const cuuint64_t sb = d.B > 1 ? (cuuint64_t)st.b * 2 : (heads > 1 ? sh * heads : row * d.S);
  if (sh == 0 || sb == 0) { set_error("zero head/batch strides are not supported by the tcgen05 kernel"); return PBS_ERR_LAYOUT; }
  const cuuint64_t dims[4] = {(cuuint64_t)d.D, (cuuint64_t)d.S, (cuuint64_t)heads, (cuuint64_t)d.B};
  const cuuint64_t strides[3] = {row, sh, sb};
  const cuuint32_t box[4] = {64, 128, 1, 1}, estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, dt == PBS_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r); return PBS_ERR_CUDA; }
  return PBS_OK;
}

template <typename K>
int launch_regs(K* kernel) {
  cudaFuncAttributes at;
  return cudaFuncGetAttributes(&at, kernel) == cudaSuccess ? at.numRegs : -1;
}

template <int DT, int D>
int run_tc(const Dims& d, const void* q, Strides qs, const KvSource& kv, const int32_t* idx,
           const uint32_t* list, const int32_t* count, void* out, Strides os, int32_t* status, int32_t* queue,
           const pbs_out_replicas_t* replicas, cudaStream_t st) {
  CUtensorMap mq, mk, mv;
  int rc = make_map(&mq, DT, q, d, d.Hq, qs);
  if (!rc) rc = make_map(&mk, DT, kv.k, d, d.Hq / kv.group, kv.ks);
  if (!rc) rc = make_map(&mv, DT, kv.v, d, d.Hq / kv.group, kv.vs);
  if (rc) return rc;
  Params p;
  p.idx = idx; p.kv_group = kv.group; p.list = list; p.count = count; p.out = out; p.os = os;
  p.Hq = d.Hq; p.S = d.S; p.G = (d.S + 255) / 256; p.T = (d.S + 127) / 128;
  p.bs = d.bs;
  p.scale_log2e = (float)(1.4426950408889634 / sqrt((double)d.D));
  p.status = status;

  p.n_extra = replicas ? replicas->count : 0;
  for (int x = 0; x < PBS_MAX_OUT_REPLICAS; ++x) p.extra_out[x] = x < p.n_extra ? replicas->out[x] : nullptr;
  p.wait_ns = g_wait_ns.load(std::memory_order_relaxed);
  p.drop_arrive = g_drop_arrive.load(std::memory_order_relaxed);
  const int sm_count = device_sms();
  auto kern = queue ? attn_tc_kernel<DT, D, true> : attn_tc_kernel<DT, D, false>;
  const int smem = kSmemBytes<D>;
  cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (ce != cudaSuccess) return cuda_fail(ce, "attn_tc_kernel smem attribute");
  // The warps share out what the launch has (kRegsIssue, kRegsSoftmax): more would be waited for without an end.
  static const bool regs_fit = launch_regs(attn_tc_kernel<DT, D, true>) == kRegsLaunch && launch_regs(attn_tc_kernel<DT, D, false>) == kRegsLaunch;
  if (!regs_fit) { set_error("attn_tc_kernel was not built with %d registers a thread", kRegsLaunch); return PBS_ERR_CUDA; }
  p.queue = queue;
  p.work = make_schedule(d.B * d.Hq, p.G, sm_count);
  kern<<<queue ? p.work.ctas : entries(p.work), kThreads, smem, st>>>(mq, mk, mv, p);
  PBS_CUDA_CHECK_LAUNCH("attn_tc_kernel");
  return PBS_OK;
}

}  // namespace

void set_attn_wait(unsigned long long wait_ns, int drop_arrive) {
  g_wait_ns.store(wait_ns ? wait_ns : 2000000000ull, std::memory_order_relaxed);
  g_drop_arrive.store(drop_arrive < 0 ? 1 : drop_arrive, std::memory_order_relaxed);
}

bool attn_tc_supported(const Dims& d, int dt) {
  return (dt == PBS_BF16 || dt == PBS_FP16) && (d.D == 64 || d.D == 128) && (d.bs == 64 || d.bs == 128) &&
         (d.seg % 128 == 0 || (d.seg == 64 && d.bs == 64)) && (d.S + 127) / 128 <= 0xFFFF;
}

int launch_attn_tc(const Dims& d, int dt, const void* q, Strides qs, const KvSource& kv, const int32_t* idx,
                   const uint32_t* list, const int32_t* count, void* out, Strides os, int32_t* status, int32_t* queue,
                   const pbs_out_replicas_t* replicas, cudaStream_t st) {
  if (dt == PBS_BF16) {
    if (d.D == 128) return run_tc<PBS_BF16, 128>(d, q, qs, kv, idx, list, count, out, os, status, queue, replicas, st);
    return run_tc<PBS_BF16, 64>(d, q, qs, kv, idx, list, count, out, os, status, queue, replicas, st);
  }
  if (d.D == 128) return run_tc<PBS_FP16, 128>(d, q, qs, kv, idx, list, count, out, os, status, queue, replicas, st);
  return run_tc<PBS_FP16, 64>(d, q, qs, kv, idx, list, count, out, os, status, queue, replicas, st);
}

}  // namespace pbs
