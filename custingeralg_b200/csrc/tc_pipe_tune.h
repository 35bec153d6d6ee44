// What the pipeline's autotuner measures of one batch-size bin and decides from it (host only).
#pragma once

namespace tc {

constexpr int kPipeCands = 5;              // candidate tile shapes of the delta kernel
constexpr int kPipeArms = kPipeCands + 1;  // + the bin's fastest shape so far in the next bin's graph
constexpr double kMergeSlack = 0.03;

struct BinTimes {
  double per_update[kPipeArms] = {};  // ms, summed over the samples
  double batch[kPipeArms] = {};
  int n[kPipeArms] = {};  // samples

  void add(int arm, double ms, long long updates) {
    per_update[arm] += ms / (double)(updates > 0 ? updates : 1);
    batch[arm] += ms;
    n[arm] += 1;
  }
  double mean(int arm) const { return per_update[arm] / n[arm]; }
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
  // A batch in the bin's own graph (ms), and what padding it to the next bin adds; false where either was
  // not timed. The same shape is compared in both graphs, the one the bin would keep: a slower one's
  // tail hides the padding.
  bool padding(double& own, double& added) const {
    const int b = best(-1);
    if (b < 0 || n[kPipeCands] == 0) return false;
    own = batch[b] / n[b];
    added = own * (mean(kPipeCands) / mean(b) - 1.0);
    if (added < 0.0) added = 0.0;
    return true;
  }
};

// The bin whose graph serves each bin's batches: the next one's, where that adds at most kMergeSlack to a
// batch. What padding adds hardly depends on the batch, so along a chain of merged bins the steps'
// times are added up: otherwise a bin of small batches would follow larger ones, for whom each step is
// little, to a graph of a hundred times its size.
inline void merge_bins(const BinTimes* bins, int nbins, int* serve) {
  double above = 0.0;  // ms from the next bin's graph to the one that serves it
  for (int i = nbins - 1; i >= 0; --i) {
    double own = 0.0, added = 0.0;
    const bool merge = i + 1 < nbins && bins[i].padding(own, added) && added + above <= kMergeSlack * own;
    serve[i] = merge ? serve[i + 1] : i;
    above = merge ? above + added : 0.0;
  }
}

}  // namespace tc
