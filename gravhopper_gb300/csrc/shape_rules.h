// Which form of the direct sum a call gets, where that is a matter of how its targets and
// sources fill the SMs.  Plain C++, so that a host build can check the rules against
// measured times.
#pragma once

#include <stdint.h>

namespace gh {

inline int64_t div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Targets per CTA of the ordered FP64 kernel.  The time per source of the SM that holds most
// CTAs grows by 9 t + 16 with each CTA of t targets (9 FP64-pipe instructions per pair of its
// 32 lanes, and the part of the ordered sums that other CTAs do not hide), and a CTA alone on
// its SM takes no less than 13.5 t, the latency of its pair terms.  Fitted to forces of
// N = 50 to 16,000 at t = 2, 4, 5, 7 and 8: N = 1500 95 us with 5 against 114 with 4, 1800 132
// with 4 against 140 with 7, 2000 155 with 7 against 178 with 4, 3192 324 with 7 against 370
// with 8.  From 40 targets per SM on 8, the best but between 6080 and 7000 (6500 1524 us
// against 1367 with 7, 8000 1871 against 1884, 12,000 3895 against 4152).  At none of these
// sizes slower than the largest of 8, 4 and 2 that leaves two CTAs per SM.
inline int ordered_targets(int64_t nt, int num_sms) {
  if (nt >= 40LL * num_sms) return 8;
  const int forms[] = {8, 7, 5, 4, 2};
  int best = 8;
  int64_t least = -1;
  for (const int t : forms) {
    const int64_t per_sm = div_up(div_up(nt, t), num_sms);
    const int64_t busy = 2 * per_sm * (9 * t + 16), alone = 27 * t, cost = busy > alone ? busy : alone;
    if (least < 0 || cost < least) {
      least = cost;
      best = t;
    }
  }
  return best;
}

// Whether a mixed sum of np sources on nt targets, one side short, takes tiles of 64 threads x
// 2 targets (six CTAs per SM) instead of 512 x 4 (one): tiles of 2048 targets leave SMs idle
// or the last wave of them nearly empty, small ones cost a ninth more per pair.  In units of
// 0.6 us: 120 per unit (tile x chunk of 512 sources) of the busiest CTA with large tiles, 50
// with small ones, and 1 per CTA that shares a large tile, whose partial sums one CTA adds.
// Large / small tiles: 100 targets x 100,000 sources 239 / 99 us, 4000 x 300,000 628 / 638,
// 50,000 targets x 1000 sources 101 / 60, 200,000 x 1500 166 / 192, 1,000,000 x 2048 860 / 924.
inline bool small_tiles(int64_t np, int64_t nt, int num_sms) {
  if (nt > 4096 && np > 2048) return false;
  const int64_t chunks = div_up(np, 512), large = div_up(nt, 2048), small = div_up(nt, 128);
  const int64_t sharing = div_up(num_sms, large) < chunks ? div_up(num_sms, large) : chunks;
  return 50 * div_up(small * chunks, 6LL * num_sms) <= 120 * div_up(large * chunks, num_sms) + sharing;
}

}  // namespace gh
