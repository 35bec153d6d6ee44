// What the pipeline's autotuner measures of one batch-size bin and decides from it (host only).
#pragma once

namespace tc {

constexpr int kPipeCands = 5;              // candidate tile shapes of the delta kernel
constexpr int kPipeArms = kPipeCands + 1;  // + the bin's fastest shape so far in the next bin's graph
constexpr double kMergeSlack = 1.03;

struct BinTimes {
  double ms[kPipeArms] = {};  // per update, summed over the samples
  int n[kPipeArms] = {};      // samples

  void add(int arm, double ms_per_update) {
    ms[arm] += ms_per_update;
    n[arm] += 1;
  }
  double mean(int arm) const { return ms[arm] / n[arm]; }
  // The arm to run next: the first of those with the fewest samples.
  int next(int arms) const {
    int a = 0;
    for (int j = 1; j < arms; ++j)
      if (n[j] < n[a]) a = j;
    return a;
  }
  // The fastest shape in the bin's own graph; `untuned` where none was timed.
  int best(int untuned) const {
    int b = -1;
    for (int j = 0; j < kPipeCands; ++j)
      if (n[j] > 0 && (b < 0 || mean(j) < mean(b))) b = j;
    return b < 0 ? untuned : b;
  }
  // Does padding to the next bin cost nothing? The same shape is compared in both graphs, the one the
  // bin would keep: a slower one's tail hides the padding.
  bool merges() const {
    const int b = best(-1);
    return b >= 0 && n[kPipeCands] > 0 && mean(kPipeCands) <= kMergeSlack * mean(b);
  }
};

}  // namespace tc
