// kernels.h — host-side launchers of the libgba kernels (one per kernel
// family; the precision mode picks the template instance).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "gba_internal.h"

namespace gba {

// LM state initialisation (per problem).
void launch_init_state(const DeviceBatch &b, cudaStream_t s);
// K0: camera tables (R, dR/dw, t, f, k1, k2) of the current parameters (a
// problem's first evaluation; K5b writes the later ones).
void launch_camera_table(const DeviceBatch &b, cudaStream_t s);
// K1 + K1c: residuals, scaled & corrected Jacobian, point blocks (chunk
// kernel) and camera blocks (camera kernel).  norms = first pass of the
// solve: unscaled column norms only.
void launch_eval_jacobian(const DeviceBatch &b, bool mixed, bool norms, cudaStream_t s);
// Jacobi scaling from the column norms of the first pass.
void launch_scale_init(const DeviceBatch &b, cudaStream_t s);
// K7: per-problem cost / gradient / |x| after a Jacobian evaluation, the
// trust-region termination tests, and the LM loop condition.
void launch_post_eval(const DeviceBatch &b, cudaStream_t s);
// K3a: damped point blocks, their FP64 inverses, Cinv g_p.
void launch_point_prepare(const DeviceBatch &b, bool mixed, cudaStream_t s);
// K3b: camera-diagonal Schur blocks, reduced rhs, block-Jacobi inverse, PCG init.
void launch_camera_schur(const DeviceBatch &b, bool mixed, cudaStream_t s);
// K3c: the off-diagonal camera-camera blocks of the explicit Schur complement.
void launch_schur_form(const DeviceBatch &b, bool mixed, cudaStream_t s);
// K4a': q = S p_k with the explicit complement (launch_schur_matvec calls it
// when the batch forms S).
cudaError_t launch_schur_spmv(const DeviceBatch &b, bool mixed, cudaStream_t s, bool pdl);
// K4 cluster form: the whole PCG of every problem in one launch, one thread
// block cluster of plan.cs CTAs per problem (mixed form, explicit Schur
// complement, problems of at most kClMaxCams cameras).
constexpr int kClThreads = 512;
constexpr int kClMaxCS = 16;
constexpr int kClMaxOwn = 64;    // cameras per CTA
constexpr int kClMaxCams = 1024; // cameras per problem
struct ClusterPlan {
  int cs = 0, n_max = 0, own_max = 0;
  int threads = 0;
  bool quad = false;
  int cache_blocks = 0;  // > 0: each CTA keeps its rows of S (this many 9x9 blocks at most) in shared memory
  size_t smem = 0;
  int above = 0, upto = 1 << 30;  // the numbers of running PCGs it is launched for: (above, upto]
  // What a captured launch carries of the plan: each field is part of the
  // graph's key (batches of equal totals may split them over their problems in
  // another way, and the shared memory is laid out by the largest problem).
  void append_to(std::vector<long long> *key) const {
    key->insert(key->end(), {cs, n_max, own_max, threads, quad, cache_blocks, (long long)smem, above, upto});
  }
};
// Chooses the cluster size, the block size and whether the rows of S stay
// in shared memory, from the batch's problems (camera ranges) and the
// explicit complement's row structure (sblk_row, nc + 1); false when the
// form does not apply or cannot be launched.
// cams_per_cta: the cameras of a problem one CTA of its cluster takes (the
// cluster size follows); 0 = the shortest estimated iteration.
// quad: the quadratic-model stopping test (gba_pcg_criterion).
// running: the problems that share the GPU (num_problems, or fewer late in a
// batch).
bool pcg_cluster_plan(const ProblemInfo *prob, int num_problems, const int32_t *sblk_row, int cams_per_cta, bool quad,
                      int running, ClusterPlan *plan);
cudaError_t launch_pcg_cluster(const DeviceBatch &b, const ClusterPlan &plan, cudaStream_t s);
// K4 cluster form of the FP64 precision: as the above, the FP64 arithmetic of
// the two-kernel PCG addition for addition (the same bits), problems whose
// rows of S fit the shared memory of a cluster.
constexpr int kC64MaxCS = 16;
constexpr int kC64MaxCams = 128;
struct Cluster64Plan {
  int cs = 0, R = 0;  // CTAs per problem, rows of S per thread of the product
  bool quad = false;
  int n_max = 0, own_max = 0, pairs_max = 0;
  size_t smem = 0;
  double clocks = 0;  // estimated clocks of the largest problem's PCG iteration
  int above = 0, upto = 1 << 30;  // the numbers of running PCGs it is launched for: (above, upto]
  void append_to(std::vector<long long> *key) const {
    key->insert(key->end(), {cs, R, quad, n_max, own_max, pairs_max, (long long)smem, above, upto});
  }
};
// quad, running: as above.
bool pcg_cluster64_plan(const ProblemInfo *prob, int num_problems, const int32_t *sblk_row, bool quad, int running,
                        Cluster64Plan *plan);
cudaError_t launch_pcg_cluster64(const DeviceBatch &b, const Cluster64Plan &plan, cudaStream_t s);
// K4 grid form: the whole PCG of one problem in one launch, one CTA per SM,
// values exchanged as tagged slots (FP64 form, explicit Schur complement).
struct GridPlan {
  int grid = 0;        // CTAs launched (the ones that register share the work)
  int cap_cols = 0;    // touched columns a CTA's shared-memory layout holds
  int cap_pairs = 0;   // (row, block) pairs of one pass of the product
  bool quad = false;
  size_t smem = 0;
  void append_to(std::vector<long long> *key) const {
    key->insert(key->end(), {grid, cap_cols, cap_pairs, quad, (long long)smem});
  }
};
// The CTAs' shares.  The units of the product: a camera's rows in the pairs
// (0,1) (2,3) (4,5) (6,7) and row 8, the first level of the camera's p.q sum.
// A row costs the camera's blocks m (off-diagonal + diagonal), a pair 2 m; the
// units are cut into P runs of about equal cost.  Units of a camera that start
// before the cost bound t, the rows before the camera costing `before` in all.
__host__ __device__ inline int units5_below(long long t, long long before, long long m) {
  if (t <= before) return 0;
  const long long r = (t - before + 2 * m - 1) / (2 * m);
  return r > 5 ? 5 : (int)r;
}
// CTA w's cost bound, of `rows` = the problem's blocks (the diagonal ones
// included): it owns the units that start in [bound(w), bound(w + 1)).
__host__ __device__ inline long long grid_bound(int w, int P, long long rows) { return ((long long)w * 9 * rows + P - 1) / P; }
// CTA w's run of `total` camera blocks or chunks of cameras: from here to w + 1's.
__host__ __device__ inline int grid_run(int w, int P, int total) { return (int)((long long)w * total / P); }
// Only a CTA that publishes something every iteration may read what the
// others publish: nothing holds a slot for a reader that no one waits for.
__host__ __device__ inline bool grid_takes_part(int units, int blocks, int chunks) { return units > 0 || blocks > 0 || chunks > 0; }
// Sizes the launch from the problem's explicit-complement structure
// (sblk_row, nc + 1, and sblk_col); false when the form does not apply (a
// batch, the mixed form, the implicit complement), when the CTAs' rows of S
// would not stay in shared memory, or when its kernel cannot be resident.
// ctas: the CTAs of the launch (one per SM at most; 0 = every SM).  quad: the
// quadratic-model stopping test (gba_pcg_criterion).
bool pcg_grid_plan(int num_problems, bool mixed, bool explicit_schur, int nc, const int32_t *sblk_row,
                   const int32_t *sblk_col, int ctas, bool quad, GridPlan *plan);
cudaError_t launch_pcg_grid(const DeviceBatch &b, const GridPlan &plan, cudaStream_t s);
// K4a-b: one PCG iteration (implicit Schur mat-vec, camera-side update).
void launch_pcg_iteration(const DeviceBatch &b, bool mixed, cudaStream_t s);
cudaError_t launch_schur_matvec(const DeviceBatch &b, bool mixed, cudaStream_t s, bool pdl);
// K4b alone (one CTA per block of kPcgBlockCams cameras).
cudaError_t launch_pcg_camera(const DeviceBatch &b, bool mixed, cudaStream_t s, bool pdl);
void launch_prof_delay(cudaStream_t s);
void point_schur_init();
// Raises a kernel's dynamic shared memory limit on the current device to at
// least `bytes`, never lowering it: the limit is process-wide, and several
// engines (the serving slots) plan and capture launches of the same kernel
// with different sizes at different times.
cudaError_t raise_smem_limit(const void *func, size_t bytes);
// Kernel attributes of the PCG kernels (once per device).
void pcg_init();
// K5: point back-substitution, model cost change, candidate points.
void launch_back_substitute(const DeviceBatch &b, bool mixed, cudaStream_t s);
// K5b: candidate cameras and their tables.
void launch_candidate_cameras(const DeviceBatch &b, cudaStream_t s);
// K2: the candidate cost.
void launch_candidate_cost(const DeviceBatch &b, cudaStream_t s);
// K6: accept / reject, trust-region radius update, termination tests.
void launch_decide(const DeviceBatch &b, cudaStream_t s);
// Copies the uploaded initial parameters into both working buffers.
void launch_sync_param_buffers(const DeviceBatch &b, cudaStream_t s);
// Gathers each problem's current parameters (the buffer its parity selects)
// into out_cam (9 per camera) / out_pt (4 per point).
void launch_gather_results(const DeviceBatch &b, double *out_cam, double *out_pt, cudaStream_t s);
// Local-BA windows: camera tables at the gathered estimate, then each
// observation's chi2 = |error|^2 (B.obs_chi2).
void launch_window_chi2(const DeviceBatch &b, const double *out_cam, const double *out_pt, cudaStream_t s);

}  // namespace gba
