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
  int most, min_rows;
  // Blocks asked for: one for every min_rows rows, up to eight; `most` beyond that, once all of them have as many. Never falls as L
  // grows, so a launch sized for L has the blocks for every shorter cache.
  CDEEP_HD int bound(int L) const {
    const int n = (L + min_rows - 1) / min_rows;
    return n < 1 ? 1 : n >= most ? most : n < kPortable ? n : kPortable;
  }
  // Rows of a block: whole row steps of 16.
  CDEEP_HD int chunk(int L) const { return (((L + bound(L) - 1) / bound(L)) + 15) / 16 * 16; }
  // Blocks that have rows; the others of the launch only take part in the cluster's barriers.
  CDEEP_HD int blocks(int L) const { return L > 0 ? (L + chunk(L) - 1) / chunk(L) : 1; }
};

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
