// The key a captured solve is replayed by: two batches of equal totals whose
// cameras are split over their problems in another way differ in nothing the
// device arrays are sized by, so every plan field a launch carries is in it.
#include <algorithm>
#include <cstdio>
#include <cstring>

#include "kernels.h"
#include "prep.h"

using namespace gba;

struct Problem {
  std::vector<int32_t> cam, pt;
  std::vector<double> obs, par;
  int nc, np;
  // groups of `size` cameras that all see the group's `points` points
  Problem(int groups, int size, int points) : nc(groups * size), np(groups * points) {
    for (int j = 0; j < np; ++j)
      for (int c = 0; c < size; ++c) cam.push_back(j / points * size + c), pt.push_back(j);
    finish();
  }
  // every pair of cameras shares a point
  explicit Problem(int cameras) : nc(cameras), np(0) {
    for (int a = 0; a < cameras; ++a)
      for (int b = a + 1; b < cameras; ++b, ++np) cam.insert(cam.end(), {a, b}), pt.insert(pt.end(), {np, np});
    finish();
  }
  void finish() {
    obs.assign(2 * cam.size(), 1.0);
    par.assign(9 * (size_t)nc + 3 * (size_t)np, 0.5);
  }
  gba_problem_view view() {
    gba_problem_view v;
    std::memset(&v, 0, sizeof v);
    v.num_cameras = nc, v.num_points = np, v.num_observations = (int)cam.size();
    v.camera_index = cam.data(), v.point_index = pt.data(), v.observations = obs.data(), v.parameters = par.data();
    return v;
  }
};

template <typename T>
static std::vector<long long> key_of(const T &plan) {
  std::vector<long long> k;
  plan.append_to(&k);
  return k;
}

// Whether the key tells a plan from the same one with a field changed.
template <typename T, typename F>
static bool told(F T::*field) {
  T a, b;
  b.*field = (F)(a.*field + (F)1);
  return key_of(a) != key_of(b);
}

int main() {
  Problem dense(40), six(6, 8, 32), ten(10, 8, 32), two(2, 8, 32);
  const gba_problem_view even[] = {dense.view(), six.view(), six.view()};
  const gba_problem_view uneven[] = {dense.view(), ten.view(), two.view()};
  PrepOptions o;
  o.schur = GBA_SCHUR_EXPLICIT;
  HostBatch a, b;
  std::string err;
  if (prepare_batch(even, 3, o, &a, &err) != GBA_OK || prepare_batch(uneven, 3, o, &b, &err) != GBA_OK)
    return std::printf("failed: %s\n", err.c_str()), 1;
  auto row_max = [](const HostBatch &h) {
    int m = 0;
    for (int c = 0; c < h.nc; ++c) m = std::max(m, h.sblk_row[c + 1] - h.sblk_row[c]);
    return m;
  };
  const bool same = a.nc == b.nc && a.np == b.np && a.no == b.no && a.nchunks == b.nchunks && a.nseg == b.nseg &&
                    a.cam_blocks == b.cam_blocks && a.nblk == b.nblk && a.nup == b.nup && a.npairs == b.npairs &&
                    row_max(a) == row_max(b);
  if (!same) return std::printf("the batches' totals differ\n"), 1;
  const bool ok = told(&ClusterPlan::cs) && told(&ClusterPlan::n_max) && told(&ClusterPlan::own_max) &&
                  told(&ClusterPlan::threads) && told(&ClusterPlan::quad) && told(&ClusterPlan::cache_blocks) &&
                  told(&ClusterPlan::smem) && told(&ClusterPlan::above) && told(&ClusterPlan::upto) &&
                  told(&Cluster64Plan::cs) && told(&Cluster64Plan::R) && told(&Cluster64Plan::quad) &&
                  told(&Cluster64Plan::n_max) && told(&Cluster64Plan::own_max) && told(&Cluster64Plan::pairs_max) &&
                  told(&Cluster64Plan::smem) && told(&Cluster64Plan::above) && told(&Cluster64Plan::upto) &&
                  told(&GridPlan::grid) && told(&GridPlan::cap_cols) && told(&GridPlan::cap_pairs) &&
                  told(&GridPlan::quad) && told(&GridPlan::smem);
  if (!ok) return std::printf("a plan field is not in the key\n"), 1;
  std::printf("ok\n");
  return 0;
}
