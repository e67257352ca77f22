// How many CTA-sized groups of items a CTA of the operator's kernels walks before it retires (host code).
//
// A long walk saves the start of CTAs; a short one fills the device where there are few groups, and leaves less of it idle at
// the end.  Launches of six waves of full walks and more always take the full walk (`most`); below, a few groups decide.
// `groups` are those of one camera, `resident` the CTAs that an SM holds.  Measured at 100 to 36 000 groups, rows of 8 to 64
// channels, fp32 and 16-bit, one to six cameras: the walk chosen takes 0.1 to 0.6 % longer than the best one on average, and
// more than 3 % longer at 34 of 1308 sizes (a count of waves that takes a half-empty one for a full one: 0.2 to 3.7 %, 270).
#pragma once

namespace dfa3d {

constexpr int kFullWaves = 6;

inline bool walks_full(long long groups, int cams, int most, int resident, int sms) {
  return (groups + most - 1) / most * cams >= (long long)kFullWaves * sms * resident;
}

// What a wave of CTAs costs: `start` once, and for every group `chain`, however few CTAs are resident, plus 8 for each that is.
struct WalkCost {
  int start, chain;
};

// The walk whose waves cost the fullest SM least.  Forward, 32 points an item: 6 cameras x 1000 queries x 8 heads 95 us at
// eight groups, 70 with this rule, 1 x 1000 29 / 15, 1 x 300 28 / 7.5.  Just past a wave (batches of several items a warp, fp16,
// 8 points): 600 batches 10.4 us at one, 11.2 at two, 920 13.0 / 14.0; fp32, unrolled, with scores takes two there, 16.0 / 15.1.
inline int walk_forward(long long groups, int cams, int most, int resident, int sms, WalkCost w) {
  if (walks_full(groups, cams, most, resident, sms)) return most;
  int best = most;
  long long least = -1;
  for (int r = most; r >= 1; --r) {
    const long long n = ((groups + r - 1) / r * cams + sms - 1) / sms, waves = n / resident, left = n % resident;
    const long long cost = waves * (w.start + r * (w.chain + 8 * resident)) +
                           (left ? w.start + r * (w.chain + 8 * left) : 0);
    if (least < 0 || cost < least) {
      best = r;
      least = cost;
    }
  }
  return best;
}

// The backward waits for its reductions and pays next to nothing for a CTA's start: one group, but two where one would leave
// a second wave about half empty (760 groups of 592: 31.3 us at one, 28.6 at two, 40.0 at four; 1400: 44.4, 51.8, 51.5), and
// from eleven waves on (8900 groups of 64 channels 4 % longer at one, 7000 batches of 4 points in two stages 3 %; 5000 batches
// are 2.4 % longer at two).
inline int walk_backward(long long groups, int cams, int most, int resident, int sms) {
  if (walks_full(groups, cams, most, resident, sms)) return most;
  const long long all = groups * cams * 20, wave = (long long)sms * resident;
  return (all > 23 * wave && all <= 31 * wave) || all > 220 * wave ? (most < 2 ? most : 2) : 1;
}

}  // namespace dfa3d
