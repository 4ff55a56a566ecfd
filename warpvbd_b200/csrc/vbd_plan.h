// Which environments of a batch a launch by domains splits over clusters.  Plain C++.
#pragma once
#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

namespace vbd {

// End of the last of `jobs`, started in their order as soon as one of `places` is free.
inline double list_schedule(const std::vector<double>& jobs, int places) {
  if (places < 1) return 1e300;
  std::priority_queue<double, std::vector<double>, std::greater<double>> busy;
  double end = 0.0;
  for (double j : jobs) {
    double at = 0.0;
    if ((int)busy.size() >= places) {
      at = busy.top();
      busy.pop();
    }
    busy.push(at + j);
    end = std::max(end, at + j);
  }
  return end;
}

// Predicted time of one launch that gives the first h environments a cluster of C blocks
// each and the others one block each.  d1, dC: durations on one block and on C, environments
// by descending d1.  Clusters are the unit the device places: a split environment's, or one
// of C single-block environments, which ends with its longest.  Without a split (h = 0) the
// blocks need no clusters, and several share an SM beyond one each.
inline double launch_time(const std::vector<double>& d1, const std::vector<double>& dC, int h,
                          int C, int clusters, int sms) {
  const int n = (int)d1.size();
  if (h == 0) {
    double sum = 0.0;
    for (double d : d1) sum += d;
    return std::max(d1[0], n > sms ? sum / sms : 0.0);
  }
  std::vector<double> jobs(dC.begin(), dC.begin() + h);
  std::sort(jobs.begin(), jobs.end(), std::greater<double>());
  for (int i = h; i < n; i += C) jobs.push_back(d1[i]);
  return list_schedule(jobs, clusters);
}

// The split count with the smallest launch time among: none, all, the most that start
// together with all the others, and `bound` (the planner's, whose estimate knows no order:
// it counts blocks that start late as if they filled the gaps).  *time: its launch time.
inline int split_count(const std::vector<double>& d1, const std::vector<double>& dC, int C,
                       int clusters, int sms, int bound, double* time = nullptr) {
  const int n = (int)d1.size();
  // h + ceil((n - h) / C) <= clusters
  int together = 0;
  while (together < n && together + 1 + (n - together - 1 + C - 1) / C <= clusters) ++together;
  int best = 0;
  double best_t = launch_time(d1, dC, 0, C, clusters, sms);
  for (int h : {bound, together, n}) {
    if (h <= 0) continue;
    // at least its jobs' total over the places: most counts end here, without a simulation
    double total = 0.0;
    for (int i = 0; i < h; ++i) total += dC[i];
    for (int i = h; i < n; i += C) total += d1[i];
    if (total >= best_t * clusters) continue;
    const double t = launch_time(d1, dC, h, C, clusters, sms);
    if (t < best_t * 0.999) {
      best_t = t;
      best = h;
    }
  }
  if (time) *time = best_t;
  return best;
}

// Blocks per cluster of a batch whose caller names none: `preferred`, or half of it and so
// on down to 2 where no cluster of the larger size can be resident, or where the smaller is
// predicted to be faster by more than the model's error (a tenth).  clusters(C): how many can
// be resident; time(C, clusters): the predicted launch time.  1 if no cluster can be.
template <class Clusters, class Time>
int pick_cluster(int preferred, Clusters clusters, Time time) {
  int best = 1;
  double best_t = 1e300;
  for (int C = preferred; C >= 2; C /= 2) {
    const int k = clusters(C);
    if (k < 1) continue;
    const double t = time(C, k);
    if (best == 1 || t < 0.9 * best_t) {
      best = C;
      best_t = t;
    }
  }
  return best;
}

}  // namespace vbd
