// Order of the attention kernel's work items; plain C++, so that the host can check it.
#pragma once

#ifdef __CUDACC__
#define PBS_HD __host__ __device__ __forceinline__
#else
#define PBS_HD inline
#endif

namespace pbs {

// Work order.  Within a head the query groups are taken in the order G-1, 0, G-2, 1, ... and a CTA
// takes two consecutive positions at a time, i.e. a long group followed by the short group that
// complements it: every such pair has the same number of key tiles (2G + 2 in the dense case), so
// all CTAs start their long group at the same time and walk up the head's key range together -- a K/V
// tile is then fetched from HBM once and served to the other CTAs from L2, instead of every CTA
// sweeping at its own position.
// The pairs rarely fill the last wave of CTAs, a pair is too coarse to share out, and where the selection is sparse
// the groups of a length differ.  So the work is a queue that CTAs draw from: first the pairs, all but those of
// the last full wave and what is left over; those are dealt out group by group, the longest of all heads left first.
// The counter of the draws has to belong to one launch alone.  The whole-path call has such a word (its scratch serves one
// call at a time and is cleared at its start); the stage call has not, because its status words may be shared by launches
// that overlap.  It starts a CTA per entry instead, in the same order, which costs a start-up an entry.
// us of a whole call with the queue / a CTA per entry / fixed pairs, 32 heads: 4 x 2048 tokens 368 / 377 / 396, 6001 sparse tokens (fp16) 346 /
// 348 / 379, 8192 of head_dim 64 478 / 481 / 535, a layer of 8192 1287 / 1295 / 1326, 32768 sparse 4337 / 4338 / 4490; 4 heads of 131072
// tokens 14.36 / 14.34 / 14.49 ms.
struct Schedule {
  int n_items, G, BH;               // query groups of all heads; groups a head; heads of all sequences
  int ctas;                         // CTAs that share the work out of a queue, at most one a SM
  int pairs;                        // entries of the queue that are pairs; the others are single groups
};
PBS_HD int entries(const Schedule& w) { return w.n_items - w.pairs; }
inline Schedule make_schedule(int BH, int G, int sms) {
  const int items = BH * G, ctas = items < sms ? items : sms;
  const int waves = items / 2 / ctas;                      // full waves of pairs
  return Schedule{items, G, BH, ctas, ctas * (items == 2 * ctas * waves ? waves : (waves > 0 ? waves - 1 : 0))};
}
// Queue entry q, its j-th item (j = 1 only for pairs); false past the end.
PBS_HD bool queue_item(const Schedule& w, int q, int j, int& bh, int& g) {
  if (q < w.pairs) {
    const int pos = 2 * q + j, r = pos % w.G;
    bh = pos / w.G;
    g = (r & 1) ? (r >> 1) : (w.G - 1 - (r >> 1));
    return true;
  }
  const int first = 2 * w.pairs;                           // positions the pairs have taken
  int k = q - w.pairs;
  if (j || k >= w.n_items - first) return false;
  // the first head left may have lost its longest and its shortest groups to the pairs: [lo, hi] remain
  const int bh0 = first / w.G, r0 = first % w.G;
  const int lo = r0 >> 1, hi = w.G - 1 - ((r0 + 1) >> 1);
  const int whole = w.BH - bh0 - 1;                        // heads after it, with all their groups
  const int above = (w.G - 1 - hi) * whole, within = (hi - lo + 1) * (whole + 1);
  if (k < above) {
    g = w.G - 1 - k / whole;
    bh = bh0 + 1 + k % whole;
  } else if ((k -= above) < within) {
    g = hi - k / (whole + 1);
    bh = bh0 + k % (whole + 1);
  } else {
    k -= within;
    g = lo - 1 - k / whole;
    bh = bh0 + 1 + k % whole;
  }
  return true;
}

}  // namespace pbs
