// How the cached rows of a (sequence, key head) pair are shared out over the blocks of its cluster. Used by the host for the size of the
// launch and by the device where the number of rows is read there, so both share out (and therefore round) identically.
#pragma once
#include <atomic>

#ifdef __CUDACC__
#define CDEEP_HD __host__ __device__
#else
#define CDEEP_HD
#endif

namespace cdeep {

constexpr int kMaxSplits = 16;  // of a pair: the largest cluster that there is
constexpr int kPortable = 8;    // the largest that every device takes

struct DecodeSplit {
  int most = 1, large_from = 0;             // blocks at most, and from how many rows on more than eight of them
  int many = 0, many_from = 1 << 30;        // from that many rows on: `many` blocks, in clusters of eight
  int waves = 0, more_from[4] = {};         // more pairs than two blocks of each fit: one block, and one more from each of these rows on
  // Blocks asked for: one for every 48 rows, up to eight; `most` beyond that. Never falls as L grows (large_from is at least eight
  // times 48), so a launch sized for L has the blocks for every shorter cache.
  CDEEP_HD int bound(int L) const {
    if (waves) return 1 + (L >= more_from[0]) + (L >= more_from[1]) + (L >= more_from[2]) + (L >= more_from[3]);
    if (L >= many_from) return many;
    if (most > kPortable && L >= large_from) return most;
    const int n = (L + 47) / 48, cap = most < kPortable ? most : kPortable;
    return n < 1 ? 1 : n < cap ? n : cap;
  }
  // Rows of a block: whole row steps of 16.
  CDEEP_HD int chunk(int L) const { return (((L + bound(L) - 1) / bound(L)) + 15) / 16 * 16; }
  // Blocks that have rows; the others of the launch only take part in the cluster's barriers.
  CDEEP_HD int blocks(int L) const { return L > 0 ? (L + chunk(L) - 1) / chunk(L) : 1; }
};

// More pairs than two blocks of each fit the device at once: c blocks a pair (a cluster; active[c - 1] of which fit) take as many waves
// as their number asks for, each as long as a block's rows and some 100 more (its start, the query, the merge); the last wave is
// shorter only down to 65 % of the others, below which its blocks have bandwidth to spare and are chains of their own.
inline DecodeSplit split_of_waves(long long pairs, const short* active) {
  DecodeSplit r;
  double waves[5];
  for (int c = 1; c <= 5; ++c) {
    const double full = static_cast<double>(pairs / active[c - 1]), last = static_cast<double>(pairs % active[c - 1]) / active[c - 1];
    waves[c - 1] = full + (last > 0 && last < 0.65 ? 0.65 : last);
  }
  r.waves = r.most = 1;
  for (int& from : r.more_from) from = 1 << 30;
  // time of L rows with c blocks: waves (L / c + 100); the next c is the first to undercut the one before
  for (int cur = 1; cur < 5;) {
    int next = 0;
    double at = 1e9;
    for (int c = cur + 1; c <= 5; ++c) {
      const double gain = waves[cur - 1] / cur - waves[c - 1] / c, cost = 100 * (waves[c - 1] - waves[cur - 1]);
      if (gain > 0 && cost / gain < at) next = c, at = cost / gain;
    }
    if (!next || at > 60000) break;
    for (int i = cur - 1; i < next - 1; ++i) r.more_from[i] = at < 1 ? 1 : static_cast<int>(at) + 1;
    r.most = cur = next;
  }
  return r;
}

// A number that is asked of the driver once per device (twice where threads come at the same time).
class DeviceNumber {
 public:
  template <typename Ask>
  int get(int device, Ask ask) {
    if (device < 0 || device >= kDevices) return ask();
    int n = known_[device].load(std::memory_order_acquire);
    if (n == 0) {
      n = ask() + 1;
      known_[device].store(n, std::memory_order_release);
    }
    return n - 1;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> known_[kDevices] = {};
};

// The largest cluster that a device holds: 16 or 13 blocks where it says so (a partition whose clusters have fewer SMs may not),
// else the eight that every device takes.
template <typename Fits>
int largest_cluster(Fits fits) {
  return fits(kMaxSplits) ? kMaxSplits : fits(13) ? 13 : kPortable;
}

}  // namespace cdeep
