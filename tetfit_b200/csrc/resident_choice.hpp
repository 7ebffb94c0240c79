// Which launches the resident CG kernels (grp_cg_resident, pcg_resident) can
// make for a system: rows a thread, warps a block, clusters.  Host rules
// without CUDA calls; what the device allows comes in through the callers'
// queries, and a choice that the device does not allow is not made.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace tf {

constexpr int kCgVals = 5;      // most values of an exchange
constexpr int kCgChunks = 10;   // 32-block chunks of a system
constexpr int kCgCluster = 16;  // most blocks of a cluster

// exchange boxes of `blocks` blocks: two sets of 16-byte records
constexpr size_t cg_box_bytes(size_t blocks) { return 2 * kCgVals * blocks * blocks * 16; }

struct ResidentChoice {
  int rows = 0;     // rows a thread, 0: no resident launch
  int warps = 0;    // warps a block
  int blocks = 0;   // blocks of the launch (grp_cg_resident: 0, as the members need)
  int cluster = 1;  // blocks of a cluster
  int entries = 0;  // matrix entries a block's shared memory holds
};

// ------------------------------------------------------------- tf_pcg_solve
constexpr int kPcgThreads = 512;
constexpr int kPcgClusterRows = 20480;

inline ResidentChoice pcg_choice(int64_t n, int blocks, int cluster, int rows, int entries) {
  ResidentChoice c;
  if (entries < 1) return c;
  const int64_t slices = (n + 31) / 32;
  c.rows = rows;
  c.cluster = cluster;
  c.entries = entries;
  // as few warps as the blocks allow, but not fewer than 8
  c.warps = std::max(8, (int)((slices + (int64_t)blocks * rows - 1) / ((int64_t)blocks * rows)));
  // clusters take all their blocks (the last ones may have no rows)
  c.blocks = cluster > 1 ? blocks : (int)((slices + (int64_t)c.warps * rows - 1) / ((int64_t)c.warps * rows));
  return c;
}

// Blocks that exchange with one another, one an SM, to 8 rows a thread.
// entries(rows): what a block's shared memory holds, 0 when the kernel cannot
// be launched.
template <typename Entries>
ResidentChoice pcg_flat(int64_t n, int sms, Entries entries) {
  for (int rows : {1, 2, 4, 8})
    if (n <= (int64_t)rows * sms * kPcgThreads) return pcg_choice(n, sms, 1, rows, entries(rows));
  return {};
}

// Clusters of 8 blocks exchange within themselves through distributed shared memory
// first, so 15 blocks instead of 148 poll one another's boxes.  An iteration
// on grid matrices takes 6.8 against 7.4 us at 27,000 rows (flat, the same with
// 30 blocks: 5.7 against 5.8 us at 15,600 rows, so small systems stay flat), 7.5
// against 8.8 at 67,650, 8.5 against 9.4 at 131,150, 8.6 against 14.3 at 162,000.
// clusters(): how many of them run at once.
template <typename Clusters, typename Entries>
ResidentChoice pcg_clustered(int64_t n, Clusters clusters, Entries entries) {
  if (n <= kPcgClusterRows) return {};
  const int blocks = 8 * clusters();
  for (int rows : {1, 2, 3})
    if (n <= (int64_t)rows * blocks * kPcgThreads) return pcg_choice(n, blocks, 8, rows, entries(rows));
  return {};
}

// ------------------------------------------------------------------- groups
constexpr int kCgResidentWarps = 16;  // most warps of a block: 128 registers a thread hold up to 8 rows
constexpr int kCgResidentRows = 8;    // most rows of a thread

// The launches for a group of members of `slices` 32-row slices each, the
// preferred one first; none when its rows do not fit one block an SM.
// entries(rows) as above; clusters(rows, entries, size): clusters of `size`
// blocks that run at once.
template <typename Entries, typename Clusters>
std::vector<ResidentChoice> group_choices(const std::vector<int64_t>& slices, int sms, bool fp32, Entries entries,
                                          Clusters clusters) {
  sms = std::min(sms, 32 * kCgChunks);
  auto blocks = [&](int64_t per) {
    int64_t g = 0;
    for (int64_t n : slices) g += (n + per - 1) / per;
    return g;
  };
  for (int64_t n : slices)
    if (n == 0) return {};
  // rows a thread: as few as keep one block an SM, and then as few warps, but
  // not fewer than 8: the exchanges of a small system stay between a few blocks
  ResidentChoice flat;
  flat.rows = 1;
  while (flat.rows <= kCgResidentRows && blocks((int64_t)kCgResidentWarps * flat.rows) > sms) flat.rows++;
  if (flat.rows > kCgResidentRows) return {};
  flat.warps = 8;
  while (flat.warps < kCgResidentWarps && blocks((int64_t)flat.warps * flat.rows) > sms) flat.warps++;
  flat.entries = entries(flat.rows);
  if (flat.entries < 1) return {};
  // Clusters (one simulation): one of 16 blocks when the rows fit it, a row a
  // thread (9^3 FP64 141 -> 120 us a solve); as many of 8 as run at once, 15 on
  // 148 SMs, when the exchange is between more than 80 blocks and the rows a
  // thread are few (FP64: up to 2, 16^3 212 -> 184 us, 24^3 285 -> 244, with 3
  // 27^3 293 -> 311; FP32: up to 4, 22^3 248 -> 211, 32^3 287 -> 258, with 7
  // 40^3 266 -> 328).  Between 17 and 80 blocks the boxes of all blocks are as
  // fast or faster (11^3 155 us against 212 with clusters of 8).
  ResidentChoice cl;
  if (slices.size() == 1) {
    const int64_t n = slices[0];
    auto fit = [&](int size, int most, int rows) {
      for (int r = 1; r <= rows && cl.rows == 0; r++) {
        const int e = entries(r), c = e > 0 ? std::min(most, clusters(r, e, size)) : 0;
        if (c < 1 || (int64_t)c * size * kCgResidentWarps * r < n) continue;
        cl.rows = r;
        cl.cluster = size;
        cl.blocks = size * c;
        cl.warps = std::max(8, (int)((n + (int64_t)cl.blocks * r - 1) / ((int64_t)cl.blocks * r)));
        cl.entries = e;
      }
    };
    if (n <= kCgCluster * kCgResidentWarps) fit(kCgCluster, 1, 1);
    else if (blocks((int64_t)flat.warps * flat.rows) > 80) fit(8, 32, fp32 ? 4 : 2);
  }
  std::vector<ResidentChoice> out;
  if (cl.rows) out.push_back(cl);
  out.push_back(flat);
  return out;
}

}  // namespace tf
