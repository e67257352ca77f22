// How the operator's kernels share the items of a launch out over the device (host code): the groups of items that a CTA
// walks before it retires, and the lanes that an item gets where a warp takes several.
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
// Waves of CTAs run into one another the more of them there are: from six of one group on, two are never slower (with scores,
// 6 x 6000 queries of 4 points, 6.1 waves, which the costs would give one: 52.9 us at one, 51.2 at two; 5000 to 9000 batches 2 to 4 %).
inline int walk_forward(long long groups, int cams, int most, int resident, int sms, WalkCost w) {
  if (walks_full(groups, cams, most, resident, sms)) return most;
  if (most == 2 && groups * cams >= (long long)kFullWaves * sms * resident) return 2;
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

// ---- kernels in which a warp takes several items (dfa3d_*_packed.cu) ---------------------------------
// Groups of C / V lanes (a row each, V channels a lane) that share an item of `lanes` lanes, each with every so-maniest point.
constexpr int groups_of_item(int C, int V, int lanes) { return V * lanes / C > 1 ? V * lanes / C : 1; }
// Lanes of an item: the next of 4, 8 and 16 from its points on ...
constexpr int lanes_of_points(int LP) { return LP <= 4 ? 4 : LP <= 8 ? 8 : 16; }
// ... or more of them in a small launch, which takes as long as one warp's chain of loads: with twice the lanes a group has
// half the points to walk.  The more it has, the larger the launch that gains by it; one point is no chain.  Where groups of
// the forward would then share the item, they add up in turns, so that its result stays the same in any launch: less to gain;
// and less where the scores come from depth bins (`bins`), whose loads come before the rows and are not shortened.
// 8 heads, us with the points' lanes / 8 / 16: 2-D, 4 points of 32 channels, forward 300 queries 4.9 / 3.8 / 3.4, 900 5.1 / 4.3 /
// 4.8 (6.6 / 5.3 / 5.3 where the map has to come from HBM), backward 8.4 / 5.4 / 4.3, 8.7 / 6.7 / 6.3; 3-D, bf16, 8 points of 64
// channels, forward 300 - / 6.4 / 5.8, 1200 - / 9.1 / 11.5, backward - / 14.9 / 10.7, - / 22.7 / 22.9.  Over 2070 sizes (60 to 2000
// queries, 2-D, 3-D, fp32 and 16-bit, 2 to 8 points of 16 to 64 channels, maps in L2 or not) 0.3 % from the best choice on
// average, more than 3 % at 85; with one line for all of them, four CTAs an SM, 3.3 % and 536.
inline int packed_lanes(int LP, int C, int V, long long items, bool backward, bool bins, int sms) {
  const int least = lanes_of_points(LP);
  int lanes = least;
  for (; lanes < 16; lanes *= 2) {
    const long long walk = (long long)LP * C, group = V * lanes;       // points a group walks: walk / group
    const long long ctas = (items * 2 * lanes + 255) / 256;
    const auto few = [&](int per_sm, int per_point, int at_most) {     // CTAs of the launch, in tenths of one an SM
      const long long limit = per_sm * group + per_point * walk;
      return 10 * ctas * group <= sms * (limit < at_most * group ? limit : at_most * group);
    };
    const bool alike = groups_of_item(C, V, 2 * lanes) == groups_of_item(C, V, least);
    const bool more = walk > group && (backward ? few(4, 7, 34)
                                       : alike ? (bins && V == 4 ? few(7, 5, 42) : few(5, 8, 60))
                                       : V == 8 ? few(5, 2, 20)        // eight channels a lane, 64 registers
                                       : bins ? few(15, 0, 15) : few(5, 5, 40));
    if (!more) break;
  }
  return lanes;
}

}  // namespace dfa3d
