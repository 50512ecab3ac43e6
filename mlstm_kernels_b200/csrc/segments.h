// When, and into how many segments, a forward of few (batch, head) units cuts its sequence.  Plain numbers, host only.
#pragma once
#include <math.h>

#include <algorithm>

namespace mlstm {

// c: 128 x 128 state tiles of a chunk boundary, over all units.  A recurrence of at most half of the SMs goes through the sequence
// in segments, and the intra-chunk kernel of a finished segment runs beside the recurrence of the next.  Estimate in
// microseconds: the intra-chunk kernel alone takes 0.013 per chunk and state tile at 8 heads 256/512 (64 tiles); one more
// segment costs 15 (drain, launch, refill).  What stays exposed is the last segment's intra-chunk work, which gives
// n = sqrt(P / 15).  Where c is more than a quarter of the SMs, the segments' recurrence has 128-column tiles, and a chunk of it takes
// 0.35 longer than in one piece, where 64-column tiles cover the SMs.  Below a gain of 8 % the extra launches are not worth their
// host time (8 heads, 49152 tokens, just above it: 808 us in five segments, 818 in one piece).
//
// With these wide tiles the intra-chunk kernel has to keep up as well, on the SMs that are left: per chunk of all units it takes
// sms / (sms - c) of its own time, which is 0.008 per unit and four output tiles and its operands at 6.55 TB/s.  Above 2.0 (against 0.95-1.2
// of the recurrence in one piece, and some slow-down of either by the other's use of the memory) nothing is gained.  Calls in us, in
// segments and in one piece, 131072 tokens in every unit, by that measure: 256/256, 16 heads, 1.92: 2201 and 2385; 64/512, 16, 1.78:
// 2040 and 2229; 256/512, 8, 1.52: 1973 and 2154; 512/1024, 2, 1.04: 1693 and 1844.  128/1024, 8, 2.06: 2508 and 2512; 64/256, 32, 2.14:
// 2422 and 2439 (65536 tokens 1195 and 1153); 64/64, 64, 2.18: 2905 and 2591; 128/512, 16, 2.20: 2613 and 2559; 128/256, 32, 2.71: 3029
// and 2841; 64/128, 64, 2.87: 3277 and 2812.  With 64-column tiles, where the recurrence leaves more of the memory's time
// unused, it is not asked: 4 heads 256/512 1140 and 1398, 32 64/128 1647 and 1827.
inline int forward_segments(long c, int NC, int units, int DHQK, int DHHV, int sms) {
  if (2 * c > sms) return 1;
  const bool wide = 4 * c > sms;
  const double P = 0.013 * (double)c * NC, slower = wide ? 0.35 * NC : 0.0;
  const int n = std::min(16, (int)lround(sqrt(P / 15.0)));
  if (n < 2) return 1;
  const double gain = P - P / n - 15.0 * (n - 1) - slower;
  if (gain <= 0.08 * (P + 1.15 * NC)) return 1;
  if (wide) {
    const double bytes = 256.0 * (2 * DHQK + 2 * DHHV) + 2.0 * DHQK * DHHV;   // q, k, v, h and the state of a chunk
    const double par = units * (0.008 * ((DHHV + 511) / 512) + bytes / 6.55e6);
    if (par * sms / (double)(sms - c) > 2.0) return 1;
  }
  return n;
}

}  // namespace mlstm
