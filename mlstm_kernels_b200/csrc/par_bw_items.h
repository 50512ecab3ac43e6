// Work items of the intra-chunk backward (chunkwise_bw_sm100.cu) and how they are dealt out to its CTAs.  Plain integers, on
// the host and the device.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define MLSTM_ITEMS_FN __host__ __device__ __forceinline__
#else
#define MLSTM_ITEMS_FN inline
#endif

namespace mlstm {

enum { PM_DV = 0, PM_DK = 1, PM_DQ = 2 };

constexpr unsigned kRunItems = 24;   // work items of a CTA at most

struct BwItems {
  int NC, DHQK, DHHV;
  int bh0;                      // first (batch, head) unit of this launch
  int maxsub;                   // most output tiles (128 columns) of an item
  int c_dv, c_dk;               // items of a chunk: deltaV's, and deltaK's and deltaQ's each
  unsigned n_items, stride;     // work items of the launch; CTAs that go through a range of them side by side
  int dx, dck, dbh;             // the stride as a step of (item of a chunk, chunk, unit)

  MLSTM_ITEMS_FN int per_chunk() const { return c_dv + 2 * c_dk; }
  // of item x of a chunk:
  MLSTM_ITEMS_FN int mode(int x) const { return x < c_dv ? PM_DV : (x < c_dv + c_dk ? PM_DK : PM_DQ); }
  MLSTM_ITEMS_FN int tile0(int x) const { return maxsub * (x < c_dv ? x : (x < c_dv + c_dk ? x - c_dv : x - c_dv - c_dk)); }
  MLSTM_ITEMS_FN int tiles(int x) const {
    const int t = ((mode(x) == PM_DV ? DHHV : DHQK) + 127) / 128 - tile0(x);
    return t < maxsub ? t : maxsub;
  }
  // slices of 64 columns in the contraction of the score and of the inter-chunk product
  MLSTM_ITEMS_FN int slices(int x) const { return ((mode(x) == PM_DV ? DHQK : DHHV) + 63) / 64; }
  // stages of the operand ring that it goes through: the score's, and of every tile the inter-chunk product's and X
  MLSTM_ITEMS_FN int stages(int x) const { return slices(x) + tiles(x) * (slices(x) + 1); }

  // ring stages of the busiest CTA (of a launch of one wave of CTAs)
  int busiest() const {
    const unsigned rounds = (n_items + stride - 1) / stride, last = n_items - (rounds - 1) * stride, gx = (unsigned)per_chunk();
    int most = 0;
    for (unsigned first = 0; first < gx && first < stride; ++first) {   // (CTAs gx apart meet the same kinds of items)
      int sum = 0;
      for (unsigned r = 0; r < rounds - (first < last ? 0 : 1); ++r) sum += stages((int)((first + r * stride) % gx));
      if (sum > most) most = sum;
    }
    return most;
  }
};

// CTA x takes every `stride`-th item; `side` of them run side by side.
inline BwItems bw_items(int units, int bh0, int NC, int DHQK, int DHHV, int maxsub, int side) {
  BwItems w{NC, DHQK, DHHV, bh0, maxsub};
  const int T_dv = (DHHV + 127) / 128, T_dk = (DHQK + 127) / 128;
  w.c_dv = (T_dv + maxsub - 1) / maxsub; w.c_dk = (T_dk + maxsub - 1) / maxsub;
  w.n_items = (unsigned)((long)w.per_chunk() * NC * units);
  w.stride = w.n_items < (unsigned)side ? w.n_items : (unsigned)side;
  const int chunks = (int)w.stride / w.per_chunk();
  w.dx = (int)w.stride % w.per_chunk(); w.dck = chunks % NC; w.dbh = chunks / NC;
  return w;
}

// One CTA per SM side by side, and up to four output tiles to an item: they share its score tile.
// Where the SM count is a multiple of the items per chunk (four, with head dims of v above 512) every CTA would meet one kind of
// item only, and kinds differ (256/1024: 24 ring stages for deltaV's, 50 for the others): a stride of one less goes through
// the kinds in turn (8 heads, 14208 tokens: 256/1024 485 and 396 us, 128/1024 320 and 258).
// A launch of less than two items per SM takes the split of its items and the stride (up to three less) that leave the busiest
// CTA the fewest ring stages, if that is a tenth fewer: a split item's parts each compute the score for themselves.  (Splitting wherever
// there are fewer items than SMs gave many of them a second round.  Kernel in us, 8 heads, so and now: 640 tokens 256/512 24.9 and
// 18.9, 192/384 22 and 16.8, 128/256 16.8 and 14.7; 512 tokens 256/256 16.8 and 14.9; 1024 tokens 256/512, two rounds of
// whole items and now of halves, 27-29 and 25.)
inline BwItems bw_plan(int units, int bh0, int NC, int DHQK, int DHHV, int sms) {
  const int T = ((DHHV > DHQK ? DHHV : DHQK) + 127) / 128;
  const BwItems whole = bw_items(units, bh0, NC, DHQK, DHHV, T < 4 ? T : 4, sms);
  if (whole.n_items >= 2u * (unsigned)sms)
    return sms % whole.per_chunk() == 0 ? bw_items(units, bh0, NC, DHQK, DHHV, whole.maxsub, sms - 1) : whole;
  BwItems best = whole;
  int most = whole.busiest();
  for (int m = whole.maxsub;; m = (m + 1) / 2) {
    for (int less = 0; less < 4 && less < sms; ++less) {
      const BwItems w = bw_items(units, bh0, NC, DHQK, DHHV, m, sms - less);
      const int b = w.busiest();
      if (10 * b < 9 * most) { most = b; best = w; }
      if (w.n_items <= w.stride) break;   // one round: the stride makes no difference
    }
    if (m == 1) return best;
  }
}

// The work items of one CTA, in the order (chunk of a unit, mode and tile group) with the stride: the CTAs of a wave go through
// neighbouring items side by side and what one chunk's modes share is in L2 while they all run.
struct BwRun {
  int x, ck, bh, left;
  MLSTM_ITEMS_FN BwRun(const BwItems& p, unsigned block, unsigned blocks) {   // (blocks: a multiple of the stride)
    const unsigned waves = blocks / p.stride, w = block / p.stride;
    const unsigned lo = (unsigned)((uint64_t)p.n_items * w / waves), hi = (unsigned)((uint64_t)p.n_items * (w + 1) / waves);
    const unsigned first = lo + (block - w * p.stride);
    left = first < hi ? (int)((hi - first + p.stride - 1) / p.stride) : 0;
    const unsigned gx = (unsigned)p.per_chunk(), r = first / gx;
    x = (int)(first - r * gx); ck = (int)(r % (unsigned)p.NC); bh = p.bh0 + (int)(r / (unsigned)p.NC);
  }
  MLSTM_ITEMS_FN void next(const BwItems& p) {
    --left;
    x += p.dx; ck += p.dck; bh += p.dbh;
    if (x >= p.per_chunk()) { x -= p.per_chunk(); ++ck; }
    if (ck >= p.NC) { ck -= p.NC; ++bh; }
  }
  MLSTM_ITEMS_FN int mode(const BwItems& p) const { return p.mode(x); }
  MLSTM_ITEMS_FN int tile0(const BwItems& p) const { return p.tile0(x); }
  MLSTM_ITEMS_FN int tiles(const BwItems& p) const { return p.tiles(x); }
  MLSTM_ITEMS_FN int slices(const BwItems& p) const { return p.slices(x); }
};

// CTAs of the launch: enough waves of them that none takes more than kRunItems
inline unsigned bw_grid(const BwItems& w) { return w.stride * ((w.n_items + w.stride * kRunItems - 1) / (w.stride * kRunItems)); }

}  // namespace mlstm
