// A batch prepared with its problems side by side on the host threads holds
// what each problem prepared alone holds, at its offsets; the error reported
// is the first failing problem's.
#include <cstdio>
#include <cstring>
#include <random>

#include "prep.h"

using namespace gba;

struct Problem {
  std::vector<int32_t> cam, pt;
  std::vector<double> obs, par;
  int nc = 0, np = 0;
  gba_problem_view view() {
    gba_problem_view v;
    std::memset(&v, 0, sizeof v);
    v.num_cameras = nc, v.num_points = np, v.num_observations = (int)cam.size();
    v.camera_index = cam.data(), v.point_index = pt.data(), v.observations = obs.data(), v.parameters = par.data();
    return v;
  }
};

template <typename T>
static bool same(const std::vector<T> &all, size_t at, const std::vector<T> &one, T add) {
  for (size_t i = 0; i < one.size(); ++i)
    if (all[at + i] != (T)(one[i] + add)) return false;
  return true;
}

int main() {
  std::mt19937 r(3);
  std::vector<Problem> pb(37);
  for (Problem &p : pb) {
    p.nc = 1 + (int)(r() % 30), p.np = (int)(r() % 900);
    for (int j = 0; j < p.np; ++j)
      for (int d = (int)(r() % 7), c0 = (int)(r() % p.nc), q = 0; q < d; ++q)
        p.cam.push_back((c0 + (int)(r() % 9)) % p.nc), p.pt.push_back(j);
    for (size_t i = p.cam.size(); i > 1; --i) {
      const size_t j = r() % i;
      std::swap(p.cam[i - 1], p.cam[j]), std::swap(p.pt[i - 1], p.pt[j]);
    }
    p.obs.resize(2 * p.cam.size());
    for (double &x : p.obs) x = (double)(r() % 1000);
    p.par.resize(9 * (size_t)p.nc + 3 * (size_t)p.np);
    for (double &x : p.par) x = (double)(r() % 100);
  }
  std::vector<gba_problem_view> v;
  for (Problem &p : pb) v.push_back(p.view());
  PrepOptions o;
  o.schur = GBA_SCHUR_EXPLICIT;
  HostBatch all;
  std::string err;
  if (prepare_batch(v.data(), (int)v.size(), o, &all, &err) != GBA_OK) return std::printf("failed: %s\n", err.c_str()), 1;
  size_t blk = 0, pair = 0, chunk = 0;
  for (size_t p = 0; p < pb.size(); ++p) {
    HostBatch one;
    if (prepare_batch(&v[p], 1, o, &one, &err) != GBA_OK) return std::printf("alone %zu: %s\n", p, err.c_str()), 1;
    const ProblemInfo &pi = all.prob[p];
    bool ok = pi.cam_count == one.nc && pi.pt_count == one.np && pi.obs_count == one.no && pi.chunk_count == one.nchunks &&
              pi.seg_count == one.nseg && (size_t)pi.chunk_begin == chunk && pi.cam_block_count == one.cam_blocks;
    ok = ok && same(all.obs_orig, pi.obs_begin, one.obs_orig, 0) && same(all.obs_cam, pi.obs_begin, one.obs_cam, pi.cam_begin) &&
         same(all.obs_pt, pi.obs_begin, one.obs_pt, pi.pt_begin) && same(all.pt_obs_begin, pi.pt_begin, one.pt_obs_begin, pi.obs_begin) &&
         same(all.obs_slot, pi.obs_begin, one.obs_slot, (uint16_t)0) && same(all.obs_seg, pi.obs_begin, one.obs_seg, (uint16_t)0) &&
         same(all.pt_orig, pi.pt_begin, one.pt_orig, 0) && same(all.seg_cam, pi.seg_begin, one.seg_cam, pi.cam_begin) &&
         same(all.seg_slot, pi.seg_begin, one.seg_slot, pi.seg_begin) && same(all.cam_seg_begin, pi.cam_begin, one.cam_seg_begin, pi.seg_begin) &&
         same(all.cam_obs_list, pi.obs_begin, one.cam_obs_list, pi.obs_begin) &&
         same(all.sblk_row, pi.cam_begin, one.sblk_row, (int32_t)blk) && same(all.sblk_col, blk, one.sblk_col, pi.cam_begin) &&
         same(all.sblk_tr, blk, one.sblk_tr, (int32_t)blk) && same(all.spair, 2 * pair, one.spair, pi.obs_begin);
    for (int c = 0; c < one.nchunks && ok; ++c)
      ok = all.chunk[chunk + c].obs_begin == one.chunk[c].obs_begin + pi.obs_begin &&
           all.chunk[chunk + c].obs_count == one.chunk[c].obs_count && all.chunk[chunk + c].problem == (int)p &&
           all.chunk[chunk + c].seg_begin == one.chunk[c].seg_begin + pi.seg_begin;
    if (!ok) return std::printf("problem %zu differs\n", p), 1;
    blk += one.nblk, pair += one.npairs, chunk += one.nchunks;
  }
  // two bad problems: the first one's error, whichever thread finds one
  for (int i = 0; i < 20; ++i) {
    pb[9].par[3] = pb[30].par[1] = 0.0 / 0.0;
    if (prepare_batch(v.data(), (int)v.size(), o, &all, &err) != GBA_ERR_NON_FINITE || err.find("problem 9: parameter 3 ") != 0)
      return std::printf("error: %s\n", err.c_str()), 1;
  }
  std::printf("ok\n");
  return 0;
}
