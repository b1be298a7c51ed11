// glp_knn_plan.h -- how a neighbour table is built: what is held on the device at a
// time (glp_knn_neighbors).  Plain C++, so that the rule and what happens when an
// allocation fails are checked on the CPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace glp {

constexpr uint32_t kKnnOperandStep = 128;  // sites of a step of the product

// Row length of the distances, in entries: whole 16-byte vectors.
inline uint32_t knn_pitch(uint32_t H) { return (H + 127u) & ~127u; }
// Operand row length in bytes: whole steps.
inline uint32_t knn_operand_pitch(uint32_t S) {
  return (S + kKnnOperandStep - 1) / kKnnOperandStep * kKnnOperandStep;
}

// The samples whose distances are held at a time, and for the Hamming metric the
// operand rows.
struct KnnPlan {
  bool tract = false, whole = false, sym = false;
  uint32_t pitch = 0;    // entries of a row of distances
  uint32_t chunk = 0;    // samples
  uint32_t bytes = 0;    // of an operand row
  uint32_t slab = 0;     // operand rows of queries, and of haplotypes, at a time
  size_t rows = 0;       // operand rows held
  size_t dist_bytes() const { return (size_t)4 * chunk * pitch; }
  size_t operand_bytes() const { return rows * bytes; }
  size_t total() const { return dist_bytes() + operand_bytes(); }
};

// The whole panel's operand is kept when it takes at most 1 GB (20,000 x 4,096: 82
// MB), else slabs of queries and of haplotypes share that.  With all distances in at
// most 1 GB (and the operand whole), only the tiles on and above the diagonal are
// computed; else chunks of 256 MB of distances.  `limit` bounds both together as far
// as 64 samples' distances and two slabs of 256 rows allow.
constexpr size_t kKnnOperandBytes = (size_t)1 << 30, kKnnSymBytes = (size_t)1 << 30,
                 kKnnChunkBytes = (size_t)256 << 20;

inline KnnPlan knn_plan(uint32_t H, uint32_t S, bool tract, size_t limit) {
  KnnPlan p;
  p.tract = tract;
  p.pitch = knn_pitch(H);
  p.bytes = knn_operand_pitch(S);
  const size_t all_dist = (size_t)2 * H * p.pitch, all_ops = tract ? 0 : (size_t)H * p.bytes;
  const size_t least = 4 * (size_t)std::min(64u, H / 2) * p.pitch;  // of distances
  const size_t ops = std::min({kKnnOperandBytes, limit / 2, limit - std::min(limit, least)});
  p.sym = all_ops <= kKnnOperandBytes && all_dist <= kKnnSymBytes && all_ops + all_dist <= limit;
  p.whole = p.sym || all_ops <= ops;
  if (!tract) {
    p.slab = p.whole ? H : (uint32_t)std::max<size_t>(256, ops / 2 / p.bytes / 256 * 256);
    p.rows = p.whole ? (size_t)H : 2 * (size_t)p.slab;
  }
  const size_t left = limit > p.operand_bytes() ? limit - p.operand_bytes() : 0;
  p.chunk = p.sym ? H / 2
                  : (uint32_t)std::min<size_t>(
                        H / 2, std::max<size_t>(64, std::min(kKnnChunkBytes, left) /
                                                        (4 * (size_t)p.pitch)));
  return p;
}

// The widest plan whose memory can be had: reserve(plan) returns 0, `no_memory`, or
// another error.  Below the caller's limit come the 256 MB that any table could be
// built in before whole panels were held, and the least.
template <class Reserve>
int knn_fitting_plan(uint32_t H, uint32_t S, bool tract, size_t limit, int no_memory,
                     Reserve reserve, KnnPlan *plan) {
  int rc = no_memory;
  size_t last = 0;
  for (const size_t at : {limit, std::min(limit, kKnnChunkBytes), (size_t)0}) {
    *plan = knn_plan(H, S, tract, at);
    if (plan->total() == last)
      continue;
    last = plan->total();
    if ((rc = reserve(*plan)) != no_memory)
      break;
  }
  return rc;
}

}  // namespace glp
