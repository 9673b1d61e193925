// The reference-layout hierarchy's coarse end on one thread-block cluster (cluster_tail.cuh).
#include "cluster_tail.cuh"

namespace ocub {

using namespace ct;

// Most pairs of cells a rank may hold of a coarsest level that is relaxed by the level kernels'
// arithmetic, one launch per colour otherwise.  A sweep costs the cluster one trip per kCtThreads pairs and
// the launches nearly nothing more.  Four V-cycles of a two-level FP32 / FP64 hierarchy, launches -> cluster
// (us): 30^3 (900 pairs) 6818 -> 4739 / 8311 -> 5800, 10x50x50 (1250) 19700 -> 16493 / 23058 -> 20532, but
// 4x64x64 (2048) 30869 -> 35251 / 36848 -> 45002, 38^3 (2166) 11444 -> 14434 / 13810 -> 18063, 50^3 (5000)
// 22280 -> 48234 / 27053 -> 62050.  The host routine's arithmetic is one CTA's work otherwise, and slower
// there at every size (50^3: 1825 ms -> 51 ms).
constexpr long long kCtDevicePairs = 3 * kCtThreads;

template <typename T>
int cluster_tail_first(const std::vector<std::array<int, 3>> &dims, bool host_coarse) {
  const int ranks = ct_max_ranks<CtPlain<T>>();
  if (!ranks) return -1;
  const auto &d = dims.back();
  const long long planes = (d[0] + ranks - 1) / ranks;
  if (!host_coarse && planes * d[1] * (d[2] / 2) > kCtDevicePairs) return -1;
  return ct_first<CtPlain<T>>(dims, 1, kCtTopCells, ranks);
}

template <typename T>
ocu_status launch_cluster_tail(const TailParams<T> &Q, bool ramp, cudaStream_t s) {
  CtParams<CtPlain<T>> P;
  std::memset(&P, 0, sizeof(P));
  std::vector<std::array<int, 3>> dims;
  for (int l = 0; l < Q.nlev; l++) dims.push_back({Q.lv[l].nx, Q.lv[l].ny, Q.lv[l].nz});
  int ranks = 1;
  const size_t bytes = ct_place(P, dims, 0, ct_max_ranks<CtPlain<T>>(), &ranks);
  for (int l = 0; l < Q.nlev; l++) {
    const TailLevel<T> &v = Q.lv[l];
    P.lv[l].k = {v.rc, v.res};
    P.lv[l].g = {v.u, v.b, v.xs, v.ys};
  }
  P.nu1 = Q.nu1;
  P.nu2 = Q.nu2;
  P.post_first = Q.post_order == 1 ? 1 : 0;
  P.coarse_iters = Q.coarse_iters;
  if (Q.coarse_order == 2) {  // symmetric: an even number, at least four
    if (P.coarse_iters % 2 == 1) P.coarse_iters++;
    if (P.coarse_iters < 4) P.coarse_iters = 4;
  }
  P.coarse_flip = Q.coarse_order == 2 ? P.coarse_iters / 2 : P.coarse_iters;
  P.host_coarse = Q.host_coarse;
  P.x.cc = Q.cc;
  P.x.unit = Q.cc.fx == 1 && Q.cc.fy == 1 && Q.cc.fz == 1;
  P.x.bc = Q.lv[0].bc;
  P.sg = boundary_signs<T>(P.x.bc);
  ct_schedule(P, ramp, ramp ? 0 : 1, Q.first_level == 0, 1LL << 62);
  return ct_launch(P, ranks, bytes, s);
}

#define INST(T)                                                                     \
  template int cluster_tail_first<T>(const std::vector<std::array<int, 3>> &, bool); \
  template ocu_status launch_cluster_tail<T>(const TailParams<T> &, bool, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace ocub
