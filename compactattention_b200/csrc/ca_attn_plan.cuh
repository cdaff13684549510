// How the attention kernels share their work out: the lengths of the 256-row kernel's units and whether they are cut
// across CTAs, and (last) the decode kernel's clusters.  Lengths are in KV steps of 128
// tokens.  Plain arithmetic on both sides: the kernel decides from the rows' counts; the host, where it knows them, by the
// same rule.  The prices and the times beside them were measured with an earlier form of the kernel and of the merge, a KV step
// of about 2.2 us; a step now takes about 2560 cycles (1.3 to 1.7 us) and the merge less too, and the prices were not taken anew.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define CA_PLAN __host__ __device__ __forceinline__
#else
#define CA_PLAN inline
#endif

namespace ca {
namespace attn {

constexpr int kSub = 64;  // tokens per TMA box / sub-block

constexpr int kMinSpanSteps = 4;           // shortest span worth a CTA of its own when units are cut
// What cutting units costs a CTA (partials, the merge), in KV steps, with up to ~8 pieces a unit; every
// further piece costs the merge about kPieceSteps more (4 units of 105 steps in 13 / 21 / 27 / 36 pieces each: 46 / 49 /
// 53 / 60 us).  Whole against cut, us: 64 units of 1-16 steps 44 / 31, 256 of them 73 / 61, 32 of ~20 37 / 32, 16 units of
// one KV head at 128K 442 / 77; units of at most 8 steps, one per SM, stay whole (27).
constexpr float kPieceSteps = 0.45f;
constexpr int kCutCostSteps = 9;
// What a unit costs beside its KV steps (Q, the first step's latency, the epilogue), in steps: the CTA with the ~29
// short units at the head of a causal first chunk of 8192 tokens ran 1.08 M cycles where one with four long units of
// the same steps ran 0.82 M, about 10,000 cycles a unit, three steps.
// us with 0 / 2 / 3 / 4: 8192 x 8192, 32/8 heads 605 / 519 / 504 / 508, 4096 x 4096, 28/4 heads 217 / 153 / 142 / 145.
constexpr int kUnitSteps = 3;

struct Units {
  int Q, tpt;      // chunk tokens; tokens per 128-row tile
  int n_pairs;     // tile pairs (units) per row
  int q_off, spb;  // tokens of the chunk region before the first query; sub-blocks per block
};

// 64-token sub-blocks of the chunk that tile pair `pair` can see.
CA_PLAN int chunk_subs(const Units& u, int pair) {
  int t_last = (2 * pair + 2) * u.tpt - 1;
  if (t_last > u.Q - 1) t_last = u.Q - 1;
  return (t_last + u.q_off) / kSub + 1;
}
CA_PLAN int unit_iters(const Units& u, int count, int pair) { return (count * u.spb + chunk_subs(u, pair) + 1) >> 1; }

// A unit's length on the line that the spans are cut from: kUnitSteps, then its KV steps.
CA_PLAN int unit_cost(const Units& u, int count, int pair) { return unit_iters(u, count, pair) + kUnitSteps; }

// Cost of the units of a row that are lane's of 32.  A row's whole cost needs 64 bits: a chunk of a million tokens with
// 128 heads to a KV head has 2^19 units of up to 2^13 steps.
CA_PLAN int lane_cost(const Units& u, int count, int lane) {
  int sum = 0;
  for (int p = lane; p < u.n_pairs; p += 32) sum += unit_cost(u, count, p);
  return sum;
}
CA_PLAN long long row_cost(const Units& u, int count) {
  long long sum = 0;
  for (int lane = 0; lane < 32; ++lane) sum += lane_cost(u, count, lane);
  return sum;
}

// Cut or whole: compare what the longest-running of g CTAs has to do.  `total` is the cost of all units, l_min and
// l_max bound a unit's.  *nc: CTAs that share the line when units are cut.  (Dealing whole units out by their number
// gave the last CTAs of a causal first chunk twice the mean work: 8192 tokens, 32/8 heads, f16 1045 us, cut by this
// rule 504 us.)
CA_PLAN bool units_are_cut(long long total, long long n_units, int l_min, int l_max, int g, int* nc_out) {
  // Cut: an equal share and the price of cutting.  With little work, fewer CTAs take longer spans (not under
  // kMinSpanSteps, and no more of them than keep share + merge of nc / n_units pieces smallest); the others leave
  // at once.
  long long nc = g;
  const long long by_work = total / kMinSpanSteps;
  const long long most = by_work > n_units ? by_work : n_units;
  if (most < nc) nc = most;
  const int best = static_cast<int>(sqrtf(static_cast<float>(total) * static_cast<float>(n_units) * (1.0f / kPieceSteps)));
  if (best < nc) nc = best > 1 ? best : 1;
  *nc_out = static_cast<int>(nc);
  const long long t_cut = total / nc + kCutCostSteps;
  // Whole: the longest unit when every unit has a CTA; equal unit counts when units are about equally long;
  // otherwise a share that ends up to a unit late.
  const long long t_whole = n_units <= g ? l_max
                            : l_min * 10LL >= l_max * 9LL ? ((n_units + g - 1) / g) * l_max
                                                          : total / g + l_max * 3LL / 4;
  // Long units: whole, the units of a KV head walk through its K and V side by side and share them in L2; pieces are
  // at different places, and with every SM busy the board holds a lower clock.  So a cut that gains little on paper loses.
  // Dense, 32/8 heads, 128 units (0.88 by this count), us cut / whole, one launch at a time; in a loop of a second
  // (power cap): 121 steps 275 / 285; 272 / 273, 249 steps 503 / 527; 577 / 543, 377 steps 765 / 768; 890 / 810, 505 steps
  // 1028 / 1000; 1204 / 1078, 761 steps 1563 / 1465; 1819 / 1612, 1017 steps 2092 / 1924; 2430 / 2128.  256 units: 241 steps
  // 946 / 1023; 1103 / 1075, 497 steps 1989 / 1956; 2284 / 2150.  The line lies where single launches break even.
  return t_cut * 100 < t_whole * (total > n_units * 512 ? 85 : 100);
}

// Whether the kernel may cut, i.e. whether the merge has to be enqueued behind it.  Where nothing is cut the merge
// still costs 2.8 us (2368 CTAs that look and leave; us with / without: 144 units of 9 steps 28.8 / 26.0, a dense call
// of 144 units of 18 to 27 steps 50.1 / 47.9).  `cap`: the most past blocks a row can have; `dense`: each row has just these.
CA_PLAN bool may_be_cut(const Units& u, int rows, int cap, bool dense, int g) {
  const int longest = unit_cost(u, cap, u.n_pairs - 1);
  if (longest <= kCutCostSteps + kUnitSteps) return false;
  const long long n_units = static_cast<long long>(rows) * u.n_pairs;
  if (dense && u.n_pairs <= 512) {  // all is known; with more units than that a row the merge is nothing
    int nc;
    return units_are_cut(rows * row_cost(u, cap), n_units, unit_cost(u, cap, 0), longest, g, &nc);
  }
  // One unit to a CTA and hardly a CTA without: only rows of unequal length make a cut pay.  Where the densities of rows
  // differ by a fifth of the past, it takes units that can have some fifty steps for that to be the price of cutting.
  return !(n_units <= g && n_units * 10 >= 9LL * g && longest <= 48);
}

// ---- decode: CTAs of a cluster that share a row of `subs` 64-token sub-blocks ----
constexpr int kMaxCluster = 8;  // 16 leaves SMs without a place for one: 1 x 131072 tokens 106 us, 8 heads; with 8 85 us
constexpr int kMinSubs = 2;     // sub-blocks a CTA of a cluster should have (1 x 1024: 5.9 us with 4, 5.1 with 2)
constexpr int kCtaSubs = 16;    // what a further wave of CTAs costs beside them, in sub-blocks (12 or less: 4 CTAs for 150 rows, 16: 2 for 304)

// Two CTAs share an SM.  Clusters sit inside a GPC, so clusters of 4 and 8 do not reach every place: 37 of 8 (every slot of
// 148 SMs) run in two waves, 32 in one.  A cluster of 8 also waits until its places in one GPC are all free, so 8 are
// only used where all fit at once (75 rows of 16384 tokens: 2 CTAs a row 93 us, 8 100).
CA_PLAN int decode_places(int cluster, int sms) { return cluster < 4 ? 2 * sms : 2 * sms * 7 / 8; }

// The cluster size with the least work in the longest-lived place: waves of CTAs x what one of them has to do.  us with
// 1 / 2 / 4 / 8 CTAs a row (* chosen): 32 rows of 32768 tokens 251 / 141 / 87 / 85*, 36 of 32768 247 / 141 / 98* / 111, 74 of
// 8192 67 / 49* / 62 / 57, 150 of 8192 92* / 114 / 103 / 103, 296 of 8192 177* / 179 / 183 / 193, 304 of 8192 219 / 197* / 186 /
// 197, 400 of 8192 245 / 233* / 239 / 261, 304 of 500 15* / 21 / 29 / 53.  (As large as keeps all CTAs resident, which it was:
// 36 rows 111, 74 rows 62, 304 rows 219.)
CA_PLAN int decode_cluster_size(long long rows, long long subs, int sms) {
  int best = 1;
  double best_cost = 0;
  for (int cs = 1; cs <= kMaxCluster && (cs == 1 || subs >= static_cast<long long>(cs) * kMinSubs); cs *= 2) {
    const long long places = decode_places(cs, sms);
    if (cs == kMaxCluster && rows * cs > places) break;
    const double cost = static_cast<double>((rows * cs + places - 1) / places) * (static_cast<double>(subs) / cs + kCtaSubs);
    if (cs == 1 || cost < best_cost) best = cs, best_cost = cost;
  }
  return best;
}

}  // namespace attn
}  // namespace ca
