// glp_width.h -- the shapes of the speculation trees, and the rule that picks a
// launch's speculation width from them.
//
// Plain C++ or CUDA: the generation kernels build their trees from these shapes
// (glp_kernels.cuh), the host side picks the width (glp_api.cu), and the rule is
// checked on the CPU.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <cmath>

namespace glp {

constexpr int kSpecNodes = 16;  // a warp's lane pairs
constexpr int kTeamNodes = 64;  // a team's of four warps
constexpr int kSpecRates = 17;  // tree i is made for a = i / 16
// Node n of a tree hangs from node parent[n], by acceptance or refusal.
struct SpecShape {
  int parent[kTeamNodes];
  bool accept[kTeamNodes];
};
constexpr SpecShape make_spec_shape(int i) {
  const double a = i == 0 ? 0.02 : i == 16 ? 0.98 : i / 16.0;
  SpecShape t{};
  double prob[kTeamNodes] = {};
  double weight[kTeamNodes][2] = {};  // of the two children, 0 once they are there
  prob[0] = 1.0;
  weight[0][0] = 1 - a;
  weight[0][1] = a;
  for (int n = 1; n < kTeamNodes; ++n) {
    int from = 0, dec = 0;
    for (int v = 0; v < n; ++v)
      for (int d = 0; d < 2; ++d)
        if (weight[v][d] > weight[from][dec]) {
          from = v;
          dec = d;
        }
    t.parent[n] = from;
    t.accept[n] = dec != 0;
    prob[n] = prob[from] * (dec ? a : 1 - a);
    weight[n][0] = prob[n] * (1 - a);
    weight[n][1] = prob[n] * a;
    // beside a refusal's child a quarter of an acceptance's is not needed: the next
    // position replaces the same slot (generation_body)
    if (!dec && weight[from][1] > 0.0)
      weight[from][1] *= 0.75;
    weight[from][dec] = 0.0;
  }
  return t;
}
// Kernels that start with 16 lanes a sample or more take trees.  Below, four nodes
// or fewer differ from the line of refusals only where a chain accepts more than 40
// % of its proposals, and the kernel without them is the faster one (3,001 x 4,000
// from codes at 8 lanes 4.39 and 4.46 ms, 10,000 x 4,096 7.36 and 7.40).
constexpr bool kSpecTree(int P) { return P >= 16; }

// The positions that a chain goes on a round, on average, at acceptance rate a with
// P lanes: the chances that the first P / 2 nodes of its tree are reached.  On a line
// of refusals (kernels without trees) an acceptance does not end the round where the
// next positions replace the same slot, each with a chance of a quarter.  For all
// widths in one pass, a node's chance from its parent's: steps[i] for 2^i lanes; line
// [i] is that of a line of a node less (a chain's first round, after its root).
constexpr int kWidths = 8;  // 1 << 0 .. 1 << 7 lanes
struct SpecShapes {
  SpecShape of[kSpecRates];
};
constexpr SpecShapes make_spec_shapes() {
  SpecShapes t{};
  for (int i = 0; i < kSpecRates; ++i)
    t.of[i] = make_spec_shape(i);
  return t;
}
inline void steps_a_round(double a, double (&steps)[kWidths], double (&line)[kWidths]) {
  static constexpr SpecShapes shapes = make_spec_shapes();
  const SpecShape &tree = shapes.of[std::min((int)(a * 16.0 + 0.5), kSpecRates - 1)];
  double chance[kTeamNodes], sum = 0.0;
  // of the line: the chances of its nodes, and of them those whose runs have
  // 4^-k left (k nodes on)
  double refusals = 0.0, runs = 0.0, refused = 1.0, last = 0.0;
  steps[0] = line[0] = 0.0;
  for (int n = 0, next = 1; n < kTeamNodes; ++n) {
    chance[n] = n == 0 ? 1.0 : chance[tree.parent[n]] * (tree.accept[n] ? a : 1.0 - a);
    sum += chance[n];
    refusals += refused;
    runs = 0.25 * runs + refused;
    refused *= 1.0 - a;
    // sum over the nodes of chance (1 + a (1/4 + 1/16 + ... to the line's end))
    const double all = refusals + a / 3.0 * (refusals - runs);
    if (n + 1 == 1 << (next - 1)) {
      steps[next] = kSpecTree(1 << next) ? sum : all;
      line[next] = last;
      ++next;
    }
    last = all;
  }
}

// What a launch is asked a width for.
struct WidthAsk {
  double rate = 0.12;     // acceptance rate, about
  uint64_t samples = 0;   // of all chunks
  double sites = 0;       // of a sample, on average
  double cycles = 0;      // of a chain, on average
  bool vq = false;
  uint32_t widest = 32;
  int sms = 0;
  double l2_bytes = 0;
  const double *resident = nullptr;  // threads that the GPU holds, for 2^i lanes
  uint32_t block_threads = 128;
};

// Speculation width of a launch: the width with the least time by a model of a
// generation, fitted to the times of every width from 4 lanes on at 2,496 points (3 to
// 40,000 samples of 3 to 8,192 sites, 5 to 100 cycles, acceptance rates 0.1 to 0.99,
// emission rows and codes), those of 50 cycles and more at rates below 0.7 with the
// most weight.  Its picks take 1.0 % longer than the best width on average, 17 % at the
// 99th percentile (at those 0.5 and 8 %); the rule before it, which knew neither the
// cycles nor what of the rows is in use at a time, 4.5 %, 60 % and at worst 125 %.
//
// A chain of C cycles has C + 1 positions.  Its first round goes over the starting
// quadruple and a line of refusals, the others as far as steps_a_round says.  While
// every sample has a group of its own, the generation lasts as long as its longest
// chain: one whose rate is off the average, a or a + min(a, kOff), whichever takes
// more rounds.  A round takes as much longer as blocks share an SM's schedulers (one
// block is a warp on each; between whole blocks kBetween of the way up to the next),
// the less the fewer sites it has, since its other parts wait more than they compute.
// Beyond the blocks that fit, groups take samples in turn: the mean chain's rounds
// times the turns, and kTail of the longest chain's.  Narrow groups stage more rows a
// lane and have fewer warps to wait for them, which costs where the rows in use exceed
// half of L2 -- those of the resident samples, not of all.  From 16 lanes on the trees
// add to every round.
//
// What it decides, in ms (width: time): 256 x 1,024 64: 0.27 (32: 0.36); 1,000 x 1,024
// 16: 0.42 (8: 0.57, 32: 0.48); 800 x 2,048 16: 0.73 (32: 0.85); 2,000 x 4,096 16: 2.16
// (8: 2.58); 5,000 x 1,024 8: 1.10 (16: 1.14); 10,000 x 4,096 8 (16: 1.9 times as long);
// 10,000 x 100 4: 0.66 (8: 0.72, 16: 0.93); 20,000 x 300 at a rate of 0.46, 20 cycles,
// 4: 0.54 (8: 0.64, 16: 0.84); 40,000 x 1,024 8 (4: 1.6 times).  2 lanes, one block an SM,
// were never the best.
constexpr double kOff = 0.513;
struct WidthCost {
  double alone;   // a round where an SM holds one block, beside 16 lanes
  double shared;  // added for each further block
  double alone_beyond, shared_beyond;  // both grow so with the rows in use beyond kFrom
};
inline double generation_time(const WidthAsk &ask, int width, const double *mean,
                              const double *mean_line, const double *off,
                              const double *off_line) {
  static constexpr WidthCost kRows[kWidths] = {{},
                                               {},
                                               {1.077, 0.315, 1.07, 0.734},
                                               {0.92, 0.404, 0.56, 0.017},
                                               {1.0, 0.382, 0, 0},
                                               {0.999, 0.412, 0, 0},
                                               {0.996, 0.485, 0, 0},
                                               {0.994, 0.474, 0, 0}};
  static constexpr WidthCost kCodes[kWidths] = {{},
                                                {},
                                                {0.959, 0.528, 0, 0},
                                                {0.952, 0.409, 0, 0},
                                                {1.0, 0.317, 0, 0},
                                                {1.145, 0.283, 0, 0},
                                                {0.987, 0.383, 0, 0},
                                                {0.977, 0.513, 0, 0}};
  constexpr double kTail = 0.372, kBetween = 0.734, kFrom = 0.476, kSpan = 0.28;  // of L2
  constexpr double kWaits = 68.201, kTrees = 27.377, kTreesOf = 50.0;             // sites
  const WidthCost cost = ask.vq ? kCodes[width] : kRows[width];
  const uint32_t P = 1u << width;
  auto rounds = [&](const double *steps, const double *line) {
    const double left = ask.cycles + 1.0 - (1.0 + line[width]);
    return left <= 0.0 ? 1.0 : 1.0 + std::max(left / steps[width], left > 0.5 ? 1.0 : left);
  };
  const double average = rounds(mean, mean_line),
               longest = std::max(average, rounds(off, off_line));
  const double groups = (double)ask.block_threads / P;
  const double blocks = std::ceil((double)ask.samples / groups);
  const double fit = std::max(1.0, ask.resident[width] / ((double)ask.block_threads * ask.sms));
  const double in_use =  // of L2, by the resident samples' rows
      std::min((double)ask.samples, fit * ask.sms * groups) * ask.sites * 16.0 / ask.l2_bytes;
  const double beyond = std::min(std::max(in_use - kFrom, 0.0), kSpan);
  const double alone = cost.alone * (1.0 + cost.alone_beyond * beyond);
  const double more = cost.shared * (1.0 + cost.shared_beyond * beyond) * ask.sites /
                      (ask.sites + kWaits);
  auto shared = [&](double held) { return 1.0 + more * (held - 1.0); };
  const double exact = blocks / ask.sms, whole = std::ceil(exact);
  const double time = whole <= fit
                          ? longest * shared(std::max(1.0, exact + kBetween * (whole - exact)))
                          : shared(fit) * (average * exact / fit + kTail * longest);
  return time * alone * (kSpecTree((int)P) ? 1.0 + kTrees / (ask.sites + kTreesOf) : 1.0);
}

inline uint32_t pick_lanes(const WidthAsk &ask) {
  const double a = ask.rate, as = std::min(a + std::min(a, kOff), 1.0);
  double mean[kWidths], off[kWidths], mean_line[kWidths], off_line[kWidths];
  steps_a_round(a, mean, mean_line);
  steps_a_round(as, off, off_line);
  uint32_t best = 8;
  double best_time = 0;
  for (int i = 2; 1u << i <= ask.widest; ++i) {
    if (ask.resident[i] <= 0)
      continue;
    const double time = generation_time(ask, i, mean, mean_line, off, off_line);
    if (best_time == 0 || time < best_time) {
      best_time = time;
      best = 1u << i;
    }
  }
  return best;
}

}  // namespace glp
