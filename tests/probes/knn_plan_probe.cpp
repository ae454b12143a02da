// Host-side sizes of the tensor-core neighbour search (test_knn_plan.py).
#include "knn.cuh"

#include <algorithm>

extern "C" {

long long probe_scratch(int n, int d, int K, int sms) {
  return static_cast<long long>(kgb::knn_tc_scratch(n, d, K, 4, sms));
}

int probe_supported(int n, int d, int K) { return kgb::knn_tc_supported(n, d, K) ? 1 : 0; }

int probe_pays(int n, int d, int K, int metric) { return kgb::knn_tc_pays(n, d, K, metric) ? 1 : 0; }

// tiles of the fold plan (0: brute force); off, skip and perm copied where room is given
int probe_fold_plan(const int* folds, int n, int d, int K, int* perm, int* off, int* skip, int* pairs) {
  const kgb::KnnFoldPlan p = kgb::knn_fold_plan(std::vector<int>(folds, folds + n), d, K, 2);
  *pairs = p.pairs;
  if (perm != nullptr) std::copy(p.perm.begin(), p.perm.end(), perm);
  if (off != nullptr) std::copy(p.off.begin(), p.off.end(), off);
  if (skip != nullptr) std::copy(p.skip.begin(), p.skip.end(), skip);
  return p.tiles;
}
}
