// glp_width.h -- the shapes of the speculation trees, and the rule that picks a
// launch's speculation width from them.
//
// Plain C++ or CUDA: the generation kernels build their trees from these shapes
// (glp_kernels.cuh), the host side picks the width (glp_api.cu), and the rule is
// checked on the CPU.
#pragma once

#include <stdint.h>

#include <algorithm>

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
// P lanes: the chances that the first P / 2 nodes of its tree are reached.  For all
// widths in one pass, a node's from its parent's: steps[i] for 2^i lanes (as powers
// of a and 1 - a, node by node and width by width, they took 14 us a launch).
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
inline void steps_a_round(double a, double (&steps)[kWidths]) {
  static constexpr SpecShapes shapes = make_spec_shapes();
  const SpecShape &tree = shapes.of[std::min((int)(a * 16.0 + 0.5), kSpecRates - 1)];
  double chance[kTeamNodes], sum = 0.0, line = 0.0, refused = 1.0;
  steps[0] = 0.0;
  for (int n = 0, next = 1; n < kTeamNodes; ++n) {
    chance[n] = n == 0 ? 1.0 : chance[tree.parent[n]] * (tree.accept[n] ? a : 1.0 - a);
    sum += chance[n];
    line += refused;
    refused *= 1.0 - a;
    if (n + 1 == 1 << (next - 1)) {
      steps[next] = kSpecTree(1 << next) ? sum : line;
      ++next;
    }
  }
}

// What a launch is asked a width for.
struct WidthAsk {
  double rate = 0.12;        // acceptance rate, about
  uint64_t samples = 0;      // of all chunks
  int sms = 0;
  bool vq = false, streams = false;  // rows beyond half of L2
  uint32_t widest = 32;
  const double *resident = nullptr;  // threads, for 2^i lanes
  uint32_t block_threads = 128;
};

// Speculation width for N samples at acceptance rate a.  A generation lasts as
// long as its longest chain while every sample has a group of its own, so the
// rule compares, for each width, the rounds of a chain whose rate is off the
// average, a or a' = a + min(a, 0.12), whichever goes on fewer positions a round,
// times what a warp's round costs at the warps a scheduler holds.  Measured
// (1,024 sites, a = 0.12, times of a generation kernel relative to one warp a
// scheduler): 1.44 at two, 2.0 at three, beyond that in proportion (whole blocks of
// four warps, so the steps are at multiples of the SM count).  Narrow groups stage
// more rows a lane and read a row for fewer evaluations: at 4 lanes 1.25, on VQ
// codes 1.5, and where the rows exceed half of L2 1.9 (measured against 8 lanes 1.5
// to 2.2: 20,000 x 512 at 8 lanes 1.65 ms, 4: 2.37; 15,000 x 2,048 4.66 and 8.28;
// 40,000 x 100, whose rows stay, 2.36 and 2.02); at 2 lanes, one block an SM, 2.7;
// at 8 lanes 1.05, and 1.1 for such rows (2,000 x 4,096 2.65 ms, 16: 2.35); on VQ
// codes, whose table reads conflict more in a wide group, 1.15 from 32.  The widths
// this picks, against others: 256 samples 64 lanes 0.27 ms (32: 0.36, 8: 0.55),
// 1,000 samples 16 lanes 0.55 (0.76; 32: 0.64), 1,500 x 2,048 8 lanes 1.07 (16:
// 1.14), 2,500 x 2,048 16 lanes 1.42 (8: 1.51), 3,001 x 4,000 from codes 16 lanes
// 3.47 (8: 3.68; 32: 4.52), 10,000 samples 8 lanes 2.05 (16: 2.49).
// 64 and 128 lanes are teams of two and four warps, for one chunk alone.  They are
// picked while every warp has a scheduler of its own: 152 x 1,024 128 lanes 0.237 ms
// (32: 0.369), 300 64 lanes 0.281 (0.355), 400 32 lanes 0.353.
inline double lane_round_cost(uint32_t P, bool vq, bool streams) {
  switch (P) {
    case 2: return 2.7;
    case 4: return vq ? 1.5 : streams ? 1.9 : 1.25;
    case 8: return streams ? 1.1 : 1.05;
    case 16: return 1.0;
    default: return vq ? 1.15 : 1.0;
  }
}

inline uint32_t pick_lanes(const WidthAsk &ask) {
  const double a = ask.rate, as = std::min(a + std::min(a, 0.12), 1.0);
  double mean[kWidths], off[kWidths];
  steps_a_round(a, mean);
  steps_a_round(as, off);
  uint32_t best = 8;
  double best_time = 0;
  for (int i = 1; 1u << i <= ask.widest; ++i) {
    if (ask.resident[i] <= 0)
      continue;
    const uint32_t P = 1u << i;
    const double consumed = std::min(mean[i], off[i]);
    const uint64_t per_block = ask.block_threads / P;
    const uint64_t blocks = (ask.samples + per_block - 1) / per_block;
    // blocks an SM holds at a time, and for one warp a scheduler in each
    const double most = std::max(1.0, ask.resident[i] / ((double)ask.block_threads * ask.sms));
    const double held = (double)((blocks + ask.sms - 1) / ask.sms);
    auto warps_cost = [](double w) { return w <= 1 ? 1.0 : w <= 2 ? 1.44 : w * (2.0 / 3.0); };
    const double a_block = ask.block_threads / 128.0;  // warps a scheduler
    const double warps = held <= most
                             ? warps_cost(held * a_block)
                             : warps_cost(most * a_block) * ((double)blocks / ask.sms) / most;
    const double time = warps * lane_round_cost(P, ask.vq, ask.streams) / consumed;
    if (best_time == 0 || time < best_time * 0.98) {
      best_time = time;
      best = P;
    }
  }
  return best;
}

}  // namespace glp
