// k_pcg_cluster64.cu — the whole FP64 PCG of a problem in one launch, one
// thread block cluster per problem (explicit Schur complement).
//
// What bounds a small problem's FP64 PCG is neither memory nor the FP64
// pipe's rate but the chain of one iteration: GB300 issues an FP64 warp
// instruction every 64 clocks per SM sub-partition (a dependent one no
// sooner, whatever the active lanes; a predicated-off one holds the pipe as
// long, hence the uniform loops below), so the iteration's ~45 dependent
// FP64 operations take about 1.5 us, and every exchange between SMs comes on
// top.  The grid form (k_pcg_grid.cu) pays three exchanges through L2 per
// iteration (0.4-1.3 us each); the two-kernel form of a batch pays two kernel
// boundaries and iterates until its slowest problem ends.  Here a cluster of
// cs <= 16 CTAs keeps its problem's rows of S in shared memory and exchanges
// through distributed shared memory between hardware cluster barriers (about
// 400 clocks each):
//   A. q = S p for the rows the CTA owns, each row's block dots summed by the
//      pairwise tree; each row's p_i q_i is stored into every CTA, q_i into
//      the CTA that updates the coordinate;              cluster barrier
//   B. every CTA: the cameras' p.q, alpha; x, r, z = M r of the camera
//      blocks (8 cameras) the CTA owns, each block's r.z, r.r (and
//      x.(v + r) when the stopping test uses it) to every CTA;
//                                                          cluster barrier
//   C. every CTA: the blocks' sums, the stopping test, beta (one warp), while
//      the other warps fetch z of the columns the CTA's rows touch; then
//      p = z + beta p.
// Measured (us per PCG iteration, local windows and rings, the grid form with
// counter barriers -> this one): 8 cameras 5.1 -> 3.4, 16 cameras 5.6 -> 4.0,
// 23 cameras 5.6 -> 4.1, 39 cameras 6.2 -> 5.5.  Batches (the PCG of one LM
// iteration, two-kernel form -> this one): 16 windows of 5-40 cameras 8.3 ->
// 2.1 ms, 48 windows 8.8 -> 2.6 ms, 200 windows 18.6 -> 8.5 ms.
// The sums are the two-kernel form's and the grid form's, addition for
// addition (kernels.cuh's trees; a butterfly level whose upper half holds
// only zeros is left out, which changes no nonzero sum), so a problem gets
// the same bits in all three forms, alone and in any batch, for any cluster
// size and any R.
// The only waits are the hardware's cluster barriers, which every CTA of a
// cluster reaches the same number of times: all decisions come from the
// same values.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "kernels.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace gba {

namespace {

constexpr int kC64Threads = 256;
constexpr int kC64Warps = kC64Threads / 32;
constexpr int kC64Slot = 96;  // threads per camera block in the update (3 warps)
constexpr int kC64Own = kC64Threads / kC64Slot;  // camera blocks a CTA updates, at most
constexpr int kC64Coords = 9 * kPcgBlockCams;
constexpr int kC64MaxBlocks = kC64MaxCams / kPcgBlockCams;
constexpr double kC64GridClocks = 11300.0;  // estimated iteration from which one problem takes the grid form
constexpr int kC64Levels = 8;  // levels of the pairwise tree (rows of up to kC64MaxCams + 1 blocks)
static_assert(kC64Coords <= kC64Slot && kC64Slot % 32 == 0, "a camera block's coordinates fit three whole warps");
static_assert(kC64MaxBlocks <= 16, "half a warp holds one quantity of every block");

// Shared memory of a CTA, the same on the host and the device.  pairs: the
// most (unit, block) pairs a CTA owns, a unit being R rows of a camera (one
// row for R = 0).
struct C64Layout {
  size_t sval, pd, p, zc, pq, csum, blkv, qv, zo, uoff, pass, pcol, ldst, total;
};
__host__ __device__ inline size_t c64_align(size_t x) { return (x + 15) & ~size_t(15); }
__host__ __device__ inline C64Layout c64_layout(int R, int n, int own_blocks, int pairs) {
  C64Layout l;
  size_t o = 0;
  const size_t oc = kC64Coords * (size_t)own_blocks;
  const size_t rows = R > 0 ? R : 1;
  l.sval = o, o = c64_align(o + 8 * 9 * rows * pairs);        // the owned rows of S, by pair
  l.pd = o, o = c64_align(o + (R > 0 ? 8 * rows * pairs : 0));  // block dots, [row of the unit][pair]
  l.p = o, o = c64_align(o + 8 * 9 * (size_t)n);              // the direction (the touched columns)
  l.zc = o, o = c64_align(o + 8 * 9 * (size_t)n);             // z of the touched columns
  l.pq = o, o = c64_align(o + 8 * 9 * (size_t)((n + 7) & ~7));  // every row's p_i q_i (stored by its owner)
  l.csum = o, o = c64_align(o + 8 * (size_t)n);               // every camera's p.q
  l.blkv = o, o = c64_align(o + 8 * 9 * 16);    // r.z, r.r, x.(v + r) of every block's three warps (stored by its owner)
  l.qv = o, o = c64_align(o + 8 * oc);          // q of the owned coordinates (stored by the row's owner)
  l.zo = o, o = c64_align(o + 8 * oc);          // z of the owned coordinates (read by the others)
  l.uoff = o, o = c64_align(o + 4 * (9 / rows * n + 1));
  l.pass = o, o = c64_align(o + (R > 0 ? 0 : 4 * (9 * (size_t)n + 1)));  // R = 0: each pass's first row, its tree levels << 16
  l.pcol = o, o = c64_align(o + (R > 0 ? 2 : 4) * (size_t)pairs);  // column camera of each pair (R = 0: c64_meta)
  l.ldst = o, o = c64_align(o + (R > 0 ? 2 * (size_t)pairs : 0));  // the tree's additions, level by level
  l.total = o;
  return l;
}

// Units of camera c (of U units, each costing its m blocks) before the cost
// bound t, the units before the camera costing `before` in all.
__host__ __device__ inline int units_below(int t, int before, int m, int U) {
  if (t <= before) return 0;
  const int r = (t - before + m - 1) / m;
  return r > U ? U : r;
}

// R = 0, what a pass needs of a pair: the column camera (8 bits), the tree
// levels in which its block takes another's sum (5: block v takes block v + s
// while v is a multiple of 2 s), whether it is its row's first block (1), the
// row (among the CTA's).
static_assert(kC64MaxCams <= 256, "a column camera in 8 bits");
__device__ __forceinline__ uint32_t c64_meta(int col, int v, int m, int row) {
  uint32_t mask = 0;
  for (int l = 0; l < 5; ++l)
    if ((v & ((2 << l) - 1)) == 0 && v + (1 << l) < m) mask |= 1u << l;
  return (uint32_t)col | mask << 8 | (v == 0 ? 1u << 13 : 0u) | (uint32_t)row << 16;
}

// Shared memory of another CTA of the cluster.
template <typename T>
__device__ __forceinline__ T *peer(T *local, int rank) {
  return cg::this_cluster().map_shared_rank(local, rank);
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace

// R > 0: the product by threads of R rows of a block each, the rows' trees
// through shared memory (the most work per FP64 instruction).  R = 0: by
// warps, the lanes over a row's blocks (several rows a pass where they fit,
// several passes a row where it is longer), the rows' trees by shuffles (no
// barrier, the shortest chain).
template <int R, bool QUAD>
__global__ void __launch_bounds__(kC64Threads) k_pcg_cluster64(DeviceBatch B, int cs, int n_max, int own_max,
                                                              int pairs_max, int above, int upto) {
  constexpr int kRows = R > 0 ? R : 1;
  constexpr int U = 9 / kRows;  // units per camera
  extern __shared__ __align__(16) unsigned char c64_smem[];
  __shared__ int s_ua, s_ub, s_lo, s_hi, s_stop, s_good, s_npass;
  __shared__ int lbeg[kC64Levels + 1], lcur[kC64Levels];
  __shared__ int blk_own[kC64MaxBlocks], blk_off[kC64MaxBlocks];
  __shared__ double sc[3], s_inv_rz, chs[4];
  __shared__ double rv[kC64Threads];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned full = 0xffffffffu;
  const int rank = cs > 1 ? (int)cg::this_cluster().block_rank() : 0;
  // (the count of running PCGs that K3b left; the other shape takes this one)
  const int running = B.status[3];
  if (running <= above || running > upto) return;
  const int prob = B.prob_order[blockIdx.x / cs];  // the longest first: the short ones fill in behind
  LMState *L = B.lm + prob;
  // uniform over the cluster: every CTA reads the state before its first
  // barrier, and rank 0 changes it only after the last one
  if (!(L->active && L->pcg_active)) return;
  const ProblemInfo pi = B.prob[prob];
  const int n = pi.cam_count, c0 = pi.cam_begin, nblk = pi.cam_block_count;
  const int r0 = B.sblk_row[c0];

  const C64Layout lay = c64_layout(R, n_max, own_max, pairs_max);
  double *sval = reinterpret_cast<double *>(c64_smem + lay.sval);
  double *pd = reinterpret_cast<double *>(c64_smem + lay.pd);
  double *p = reinterpret_cast<double *>(c64_smem + lay.p);
  double *zc = reinterpret_cast<double *>(c64_smem + lay.zc);
  double *pqb = reinterpret_cast<double *>(c64_smem + lay.pq);
  double *csum = reinterpret_cast<double *>(c64_smem + lay.csum);
  double *blkv = reinterpret_cast<double *>(c64_smem + lay.blkv);
  double *qvb = reinterpret_cast<double *>(c64_smem + lay.qv);
  double *zo = reinterpret_cast<double *>(c64_smem + lay.zo);
  int *uoff = reinterpret_cast<int *>(c64_smem + lay.uoff);
  int *pass_j = reinterpret_cast<int *>(c64_smem + lay.pass);
  unsigned short *pcol = reinterpret_cast<unsigned short *>(c64_smem + lay.pcol);  // R > 0
  uint32_t *meta = reinterpret_cast<uint32_t *>(c64_smem + lay.pcol);              // R = 0
  unsigned short *ldst = reinterpret_cast<unsigned short *>(c64_smem + lay.ldst);

  // ---- ownership -------------------------------------------------------------
  // product: the problem's units in cs runs of about equal cost (their
  // blocks); update: its camera blocks in cs runs
  if (t == 0) s_ua = 0, s_ub = 0, s_lo = n, s_hi = -1;
  if (t <= kC64Levels) lbeg[t] = 0;
  // what no camera, block or warp stores stays zero
  for (int i = t; i < 9 * ((n + 7) & ~7); i += kC64Threads) pqb[i] = 0.0;
  for (int i = t; i < 9 * 16; i += kC64Threads) blkv[i] = 0.0;
  if (t < nblk) {
    const int own = ((t + 1) * cs - 1) / nblk;  // block t lies in that CTA's run
    blk_own[t] = own;
    blk_off[t] = kC64Coords * (t - own * nblk / cs);  // its first coordinate there
  }
  __syncthreads();
  const int wtot = B.sblk_row[c0 + n] - r0 + n;
  auto before_of = [&](int c) { return B.sblk_row[c0 + c] - r0 + c; };
  {
    const int ta = (rank * U * wtot + cs - 1) / cs, tb = ((rank + 1) * U * wtot + cs - 1) / cs;
    int a = 0, b = 0;
    for (int c = t; c < n; c += kC64Threads) {
      const int before = before_of(c), m = before_of(c + 1) - before;
      a += units_below(ta, U * before, m, U);
      b += units_below(tb, U * before, m, U);
    }
    if (a) atomicAdd(&s_ua, a);
    if (b) atomicAdd(&s_ub, b);
  }
  const int kb0 = rank * nblk / cs, kb1 = (rank + 1) * nblk / cs;
  __syncthreads();
  const int ua = s_ua, nu = s_ub - ua;
  auto unit_before = [&](int u) {  // pairs of the problem's units before u
    const int c = u / U;
    if (c >= n) return U * wtot;
    return U * before_of(c) + (u - U * c) * (before_of(c + 1) - before_of(c));
  };
  const int wa = unit_before(ua);
  for (int j = t; j <= nu; j += kC64Threads) uoff[j] = unit_before(ua + j) - wa;
  __syncthreads();
  const int np = uoff[nu];
  if (R == 0) {
    // the warps' passes: as many whole rows as fit the lanes, or one longer
    // row in runs of 32 blocks
    if (t == 0) {
      int c = 0, j = 0;
      while (j < nu) {
        const int e0 = uoff[j], j0 = j++;
        int m = uoff[j] - e0;  // the longest row
        while (j < nu && uoff[j + 1] - e0 <= 32) m = max(m, uoff[j + 1] - uoff[j]), ++j;
        pass_j[c++] = j0 | (m > 1 ? 32 - __clz(m - 1) : 0) << 16;
      }
      pass_j[c] = nu;
      s_npass = c;
    }
  } else {
    // the tree's additions per level, and where each level's list begins
    for (int j = t; j < nu; j += kC64Threads) {
      const int m = uoff[j + 1] - uoff[j];
      for (int l = 0; (1 << l) < m; ++l) atomicAdd(&lbeg[l], tree_adds(m, 1 << l));
    }
    __syncthreads();
    if (t == 0) {
      int o = 0;
      for (int l = 0; l < kC64Levels; ++l) {
        const int c = lbeg[l];
        lbeg[l] = lcur[l] = o;
        o += c;
      }
      lbeg[kC64Levels] = o;
    }
    __syncthreads();
  }
  // the pairs: column camera, the unit's rows of the block, the additions
  // (their order within a level is free: each is a sum of its own)
  const double *vals = reinterpret_cast<const double *>(B.sblk_val);
  const double *Sii = reinterpret_cast<const double *>(B.cam_Sii);
  for (int j = warp; j < nu; j += kC64Warps) {
    const int u = ua + j, c = u / U, q0 = kRows * (u - U * c), e0 = uoff[j], m = uoff[j + 1] - e0;
    const int rr0 = B.sblk_row[c0 + c];
    int lo = c, hi = c;
    for (int v = lane; v < m; v += 32) {
      const int col = v < m - 1 ? B.sblk_col[rr0 + v] - c0 : c;
      if (R > 0)
        pcol[e0 + v] = (unsigned short)col;
      else
        meta[e0 + v] = c64_meta(col, v, m, j);
      lo = min(lo, col), hi = max(hi, col);
    }
    lo = __reduce_min_sync(full, lo), hi = __reduce_max_sync(full, hi);
    if (lane == 0) atomicMin(&s_lo, lo), atomicMax(&s_hi, hi);
    for (int i = lane; i < 9 * kRows * m; i += 32) {
      const int v = i / (9 * kRows), el = 9 * q0 + (i - 9 * kRows * v);
      sval[9 * kRows * e0 + i] = v < m - 1 ? vals[81 * (size_t)(rr0 + v) + el] : Sii[81 * (size_t)(c0 + c) + el];
    }
    if (R > 0)
      for (int l = 0; (1 << l) < m; ++l) {
        const int na = tree_adds(m, 1 << l);
        int base = lane == 0 ? atomicAdd(&lcur[l], na) : 0;
        base = __shfl_sync(full, base, 0);
        for (int k = lane; k < na; k += 32) ldst[base + k] = (unsigned short)(e0 + (2 << l) * k);
      }
  }
  // the update's coordinate of this thread (coordinate m of an owned camera
  // block in the lanes of three warps): its state stays in registers
  const int u_slot = t / kC64Slot, u_m = t - kC64Slot * u_slot, u_q = u_m % 9;
  const int u_blk = kb0 + u_slot;
  const bool u_in = u_slot < kC64Own && u_blk < kb1;  // uniform over the slot's three warps
  const int u_cams = u_in ? min(kPcgBlockCams, n - kPcgBlockCams * u_blk) : 0;
  const bool u_lead = u_in && u_m < 9 * u_cams;
  const bool u_warp = 32 * (warp - 3 * u_slot) < 9 * u_cams;  // the warp holds coordinates
  const int u_oc = kC64Coords * u_slot + u_m, u_i = kC64Coords * u_blk + u_m;
  const size_t u_g = 9 * (size_t)c0 + (u_lead ? u_i : 0);
  double ux = 0.0, ur = 0.0, uz = 0.0, uv = 0.0, um[9];
  if (u_lead) {
    ux = B.pcg_x[u_g], ur = B.pcg_r[u_g], uz = B.pcg_z[u_g], uv = B.pcg_v[u_g];
#pragma unroll
    for (int kk = 0; kk < 9; ++kk) um[kk] = B.cam_Minv[9 * u_g + kk];  // row u_q of the camera's block
    zo[u_oc] = uz;
    if (u_m == 0) atomicMin(&s_lo, kPcgBlockCams * u_blk), atomicMax(&s_hi, kPcgBlockCams * u_blk + u_cams - 1);
  }
  __syncthreads();
  // the touched coordinates (the columns of the owned rows and the owned
  // blocks' own): p_0 = z_0
  const int i_lo = 9 * s_lo, i_hi = 9 * (s_hi + 1);
  for (int i = i_lo + t; i < i_hi; i += kC64Threads) p[i] = B.pcg_z[9 * (size_t)c0 + i];
  int nlev = 0;
  if (R > 0)
    while (nlev < kC64Levels && lbeg[nlev + 1] > lbeg[nlev]) ++nlev;
  const int csh = 31 - __clz(cs);  // (cs is a power of two)
  // the CTA that this lane stores the update's sums into
  const int dest = lane & 15;
  double *blk_dest = cs > 1 && dest < cs ? peer(blkv, dest) : blkv;
  // q_i to the CTA that updates coordinate i
  auto push_q = [&](int i, double qv) {
    const int b = i / kC64Coords;
    double *q = qvb + blk_off[b] + (i - kC64Coords * b);
    *(cs > 1 ? peer(q, blk_own[b]) : q) = qv;
  };

  // R = 0: a pass over rows j .. j1 - 1 (pairs from e0).  A row's sum ends in
  // the lane of its first block (lead); the lanes then take (row, CTA) pairs:
  // pair x = lane stores the sum of lane src into CTA x % cs
  double *const pq_dest = cs > 1 ? peer(pqb + ua, lane & (cs - 1)) : pqb + ua;
  struct Pass {
    int j, e0, rows, levels, mask, lead, src;
    const double *s, *p, *own;
    double *dst;
    bool in;
  };
  auto pass_at = [&](int ps) {
    Pass a;
    const int pj = pass_j[ps], j1 = pass_j[ps + 1] & 0xffff;
    a.j = pj & 0xffff, a.levels = pj >> 16, a.rows = j1 - a.j;
    a.e0 = uoff[a.j];
    a.in = lane < uoff[j1] - a.e0;
    const int e = a.in ? a.e0 + lane : a.e0, row = (int)(meta[e] >> 16);
    a.mask = a.in ? (int)(meta[e] >> 8) & 31 : 0;
    a.lead = a.in && (meta[e] >> 13 & 1) ? ua + row : -1;
    a.s = sval + 9 * e, a.p = p + 9 * (int)(meta[e] & 255), a.own = p + ua + row;
    const int rr = min(a.j + (lane >> csh), j1 - 1);
    a.src = uoff[rr] - a.e0;
    a.dst = lane < a.rows << csh ? pq_dest + rr : nullptr;
    return a;
  };
  auto finish_pass = [&](double d, const Pass &a) {
    for (int l = 0; l < a.levels; ++l) {
      const double x = __shfl_down_sync(full, d, 1 << l);
      d += (a.mask >> l) & 1 ? x : 0.0;
    }
    const double pqv = *a.own * d, y = __shfl_sync(full, pqv, a.src);
    if (a.dst) *a.dst = y;
    if (a.lead >= 0) push_q(a.lead, d);
    for (int x0 = 32; x0 < a.rows << csh; x0 += 32) {  // more pairs than lanes (32 is a multiple of cs)
      const int x = x0 + lane, rr = min(a.j + (x >> csh), a.j + a.rows - 1);
      const double y2 = __shfl_sync(full, pqv, uoff[rr] - a.e0);
      if (x < a.rows << csh) pq_dest[rr] = y2;
    }
  };
  // a row of more than 32 blocks (kC64MaxCams + 1 at most): runs of 32, each
  // by a warp's tree, then the tree's levels 32, 64 and 128 over the runs
  auto long_row = [&](int j, int e0, int m0) {
    double run[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    const int nrun = (m0 + 31) / 32;
#pragma unroll
    for (int g = 0; g < 5; ++g) {
      if (g < nrun) {
        const int v = 32 * g + lane, e = e0 + min(v, m0 - 1);
        const double *sr = sval + 9 * e, *pp = p + 9 * (int)(meta[e] & 255);
        double x = 0.0;
#pragma unroll
        for (int cc = 0; cc < 9; ++cc) x = fma(sr[cc], pp[cc], x);
        run[g] = warp_pairwise_tree(v < m0 ? x : 0.0, min(32, m0 - 32 * g));
      }
    }
    run[0] += run[1];
    if (nrun > 3) run[2] += run[3];
    if (nrun > 2) run[0] += run[2];
    if (nrun > 4) run[0] += run[4];
    const double qv = __shfl_sync(full, run[0], 0), pqv = p[ua + j] * qv;
    if (lane == 0) push_q(ua + j, qv);
    if (lane < cs) pq_dest[j] = pqv;
  };
  int npass = 0;
  double a_s[9];  // the warp's first pass: its rows of S and its addresses in registers
  Pass first = {};
  int rest = warp;  // the passes from memory start here (a first pass that is a row of more than 32 blocks among them)
  if constexpr (R == 0) {
    npass = s_npass;
    if (warp < npass) {
      first = pass_at(warp);
      if (uoff[first.j + 1] - first.e0 <= 32) rest = warp + kC64Warps;
#pragma unroll
      for (int cc = 0; cc < 9; ++cc) a_s[cc] = first.in ? first.s[cc] : 0.0;
    }
  }
  const int blk_top = nblk > 8 ? 8 : nblk > 4 ? 4 : nblk > 2 ? 2 : nblk > 1 ? 1 : 0;  // the first butterfly level over the blocks

  const DeviceOptions &o = B.opt;
  double rz_k = L->rz, beta = L->beta, q0 = L->q0;
  double last_rr = L->rr, last_pq = L->pq;
  const double lim = o.pcg_tolerance * L->r0_norm;
  const long long lim2_bits = __double_as_longlong(lim * lim);
  int k = 0;
  bool linear_ok = true;
  __syncthreads();
  if (cs > 1) cluster_arrive(), cluster_wait();  // every CTA runs before any stores into it
  for (;;) {
    // ---- A. q = S p_k for the owned rows -----------------------------------
    if constexpr (R == 0) {
      if (rest > warp) {
        double d = 0.0;
#pragma unroll
        for (int cc = 0; cc < 9; ++cc) d = fma(a_s[cc], first.p[cc], d);
        finish_pass(d, first);
      }
      for (int ps = rest; ps < npass; ps += kC64Warps) {
        const int j = pass_j[ps] & 0xffff, m0 = uoff[j + 1] - uoff[j];
        if (m0 <= 32) {
          const Pass a = pass_at(ps);
          double d = 0.0;
#pragma unroll
          for (int cc = 0; cc < 9; ++cc) d = fma(a.s[cc], a.p[cc], d);
          finish_pass(d, a);
        } else {
          long_row(j, uoff[j], m0);
        }
      }
    } else {
      for (int e = t; e < np; e += kC64Threads) {
        const double *row = sval + 9 * kRows * e, *pp = p + 9 * (int)pcol[e];
        double pv[9];
#pragma unroll
        for (int cc = 0; cc < 9; ++cc) pv[cc] = pp[cc];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          double d = 0.0;
#pragma unroll
          for (int cc = 0; cc < 9; ++cc) d = fma(row[9 * r + cc], pv[cc], d);
          pd[r * np + e] = d;
        }
      }
      __syncthreads();
      for (int l = 0; l < nlev; ++l) {
        const int sp = 1 << l, lb = lbeg[l], na = lbeg[l + 1] - lb;
        for (int x = t; x < na; x += kC64Threads) {
          double *d = pd + ldst[lb + x];
          double y[kRows];
#pragma unroll
          for (int r = 0; r < kRows; ++r) y[r] = d[r * np] + d[r * np + sp];
#pragma unroll
          for (int r = 0; r < kRows; ++r) d[r * np] = y[r];
        }
        __syncthreads();
      }
      // q_i to its owner, p_i q_i here and then to the other CTAs, the threads
      // over (row, CTA)
      for (int x = t; x < kRows * nu; x += kC64Threads) {
        const int j = x / kRows, r = x - kRows * j, i = kRows * ua + x;
        const double qv = pd[r * np + uoff[j]];
        pqb[i] = p[i] * qv;
        push_q(i, qv);
      }
      if (cs > 1) {
        __syncthreads();
        for (int x = t; x < (kRows * nu) << csh; x += kC64Threads) {
          const int i = kRows * ua + (x >> csh), d = x & (cs - 1);
          if (d != rank) *peer(pqb + i, d) = pqb[i];
        }
      }
    }
    __syncwarp();
    if (cs > 1)
      cluster_arrive();
    else
      __syncthreads();
    if (warp == kC64Warps - 1 && lane == 0) s_inv_rz = recip_nr(rz_k);  // for beta, off the deciding warp's chain
    __syncwarp();
    if (cs > 1) cluster_wait();
    // ---- B. p.q: each camera's sum9_tree by four lanes (pairs, then xor 1
    // and 2, then the ninth), chunks of 32 cameras, the pairwise tree over
    // the chunks; alpha --------------------------------------------------------
    {
      double s2 = 0.0;
      for (int cb = 8 * warp; cb < n; cb += 8 * kC64Warps) {
        const int c = cb + (lane >> 2), w = lane & 3;
        const double *x9 = pqb + 9 * c;
        double x = x9[2 * w] + x9[2 * w + 1];
        const double x8 = x9[8];
        x += __shfl_xor_sync(full, x, 1);
        x += __shfl_xor_sync(full, x, 2);
        x += x8;
        if (n <= 8) {
          for (int l = n > 4 ? 16 : n > 2 ? 8 : n > 1 ? 4 : 0; l >= 4; l >>= 1) x += __shfl_xor_sync(full, x, l);
          s2 = x;
        } else if (c < n && w == 0) {
          csum[c] = x;
        }
      }
      if (n > 8) {
        __syncthreads();
        const int nch = (n + 31) / 32;
        if (warp < nch) {
          const int cnt = n - 32 * warp;
          double x = lane < cnt ? csum[32 * warp + lane] : 0.0;
          // (a level that would only add zeros is left out)
          for (int l = cnt > 16 ? 16 : cnt > 8 ? 8 : cnt > 4 ? 4 : cnt > 2 ? 2 : cnt > 1 ? 1 : 0; l > 0; l >>= 1)
            x += __shfl_xor_sync(full, x, l);
          s2 = x;
          if (nch > 1 && lane == 0) chs[warp] = x;
        }
        if (nch > 1) {
          __syncthreads();
          if (warp == 0) {
            // the pairwise tree over two to four chunks
            s2 = chs[0] + chs[1];
            if (nch == 3) s2 += chs[2];
            if (nch == 4) s2 += chs[2] + chs[3];
          }
        }
      }
      if (t == 0) {
        const long long b2 = __double_as_longlong(s2);
        sc[0] = s2, sc[1] = rz_k * recip_nr(s2);
        s_good = b2 > 0 && b2 < 0x7ff0000000000000LL;  // positive and finite
      }
      __syncthreads();
    }
    const double pq = sc[0], alpha = sc[1];
    if (s_good == 0) {  // S is not positive definite along p_k: the PCG ends with x_k
      if (k == 0) linear_ok = false;
      break;
    }
    // ---- the update of the owned camera blocks -----------------------------------
    if (u_lead) {
      ur = fma(-alpha, qvb[u_oc], ur);
      rv[t] = ur;
    }
    __syncthreads();
    if (u_in && u_warp) {
      double rz = 0.0, rr = 0.0, qx = 0.0;
      if (u_lead) {
        double zz = 0;
#pragma unroll
        for (int kk = 0; kk < 9; ++kk) zz += um[kk] * rv[t - u_q + kk];
        uz = zz;
        zo[u_oc] = uz;
        rz = ur * uz, rr = ur * ur;
      }
      // both butterflies at once: lanes 0-15 end with r.z, lanes 16-31 with
      // r.r, each lane storing its half's sum into one CTA
      const bool lo = lane < 16;
      double v = (lo ? rz : rr) + __shfl_xor_sync(full, lo ? rr : rz, 16);
      v += __shfl_xor_sync(full, v, 8);
      v += __shfl_xor_sync(full, v, 4);
      v += __shfl_xor_sync(full, v, 2);
      v += __shfl_xor_sync(full, v, 1);
      const int w = warp - 3 * u_slot;
      if (dest < cs) blk_dest[3 * ((lo ? 0 : 16) + u_blk) + w] = v;
      if constexpr (QUAD) {
        if (u_lead) {
          ux = fma(alpha, p[u_i], ux);
          qx = ux * (uv + ur);
        }
        qx = warp_sum(qx);
        if (lane < 16 && dest < cs) blk_dest[3 * (32 + u_blk) + w] = qx;
      }
    }
    __syncwarp();
    if (cs > 1) cluster_arrive();
    // x is nobody's input until the end (unless the stopping test takes it)
    if (u_lead && !QUAD) ux = fma(alpha, p[u_i], ux);
    __syncwarp();
    if (cs > 1)
      cluster_wait();
    else
      __syncthreads();
    // ---- C. warp 0: the blocks' sums (lanes 0-15 r.z, 16-31 r.r), the stopping
    // test, beta; the other warps fetch z ------------------------------------------
    if (warp == 0) {
      auto block_total = [&](const double *w3) -> double {  // over the blocks, one per lane of a half-warp
        double a = (w3[0] + w3[1]) + w3[2];
        for (int l = blk_top; l > 0; l >>= 1) a += __shfl_xor_sync(full, a, l);
        return a;
      };
      const double a = block_total(blkv + 3 * lane);
      const double rz1 = __shfl_sync(full, a, 0), rr1 = __shfl_sync(full, a, 16);
      const int k1 = k + 1;
      bool stop = false;
      if constexpr (QUAD) {
        const double qk = -__shfl_sync(full, block_total(blkv + 3 * (32 + (lane & 15))), 0);  // Q(x) = x'Sx - 2 v'x = -x.(v + r)
        const double lhs = k1 * (qk - q0), rhs = o.eta * qk;
        const bool below = qk > 0.0 ? lhs < rhs : (qk < 0.0 ? lhs > rhs : q0 > 0.0);
        if (below && k1 >= o.min_pcg_iterations) stop = true;
        q0 = qk;
      } else if (__double_as_longlong(rr1) <= lim2_bits && k1 >= o.min_pcg_iterations) {
        stop = true;  // rr1 <= lim2 (neither negative; a NaN's bits are above every number's)
      }
      if (k1 >= o.max_pcg_iterations) stop = true;
      const long long bz = __double_as_longlong(rz1) & 0x7fffffffffffffffLL;
      if (!(bz != 0 && bz < 0x7ff0000000000000LL)) stop = true;  // zero or not finite
      if (lane == 0) {
        sc[0] = rz1 * s_inv_rz;  // beta_{k+1}
        sc[1] = rz1;
        sc[2] = rr1;
        s_stop = stop ? 1 : 0;
      }
    } else {
      for (int i = i_lo + t - 32; i < i_hi; i += kC64Threads - 32) {
        const int b = i / kC64Coords;
        double *z = zo + blk_off[b] + (i - kC64Coords * b);
        zc[i] = *(cs > 1 ? peer(z, blk_own[b]) : z);
      }
    }
    __syncthreads();
    beta = sc[0];
    rz_k = sc[1];
    last_rr = sc[2];
    last_pq = pq;
    ++k;
    if (s_stop != 0) break;
    for (int i = i_lo + t; i < i_hi; i += kC64Threads) p[i] = fma(beta, p[i], zc[i]);
    __syncthreads();
  }
  // the owned coordinates' x, r, z and last direction, as the other forms
  // leave them
  if (u_lead) {
    B.pcg_x[u_g] = ux, B.pcg_r[u_g] = ur, B.pcg_z[u_g] = uz;
    if (k > 0) B.pcg_p[u_g] = p[u_i];
  }
  if (rank == 0 && t == 0) {
    L->pcg_iterations = k;
    if (!linear_ok) L->linear_ok = 0;
    if (k > 0) {
      L->beta = beta;
      L->rz = rz_k;
      L->rr = last_rr;
      L->q0 = q0;
      L->pq = last_pq;
    }
    L->pcg_active = 0;
  }
  __syncwarp();
  if (cs > 1) cluster_arrive(), cluster_wait();  // no CTA leaves before the others have read its z
}

namespace {

typedef void (*C64Kernel)(DeviceBatch, int, int, int, int, int, int);
C64Kernel c64_kernel(int R, bool quad) {
  if (quad) return R == 9 ? k_pcg_cluster64<9, true> : R == 3 ? k_pcg_cluster64<3, true> : R == 1 ? k_pcg_cluster64<1, true> : k_pcg_cluster64<0, true>;
  return R == 9 ? k_pcg_cluster64<9, false> : R == 3 ? k_pcg_cluster64<3, false> : R == 1 ? k_pcg_cluster64<1, false> : k_pcg_cluster64<0, false>;
}

void c64_config(const Cluster64Plan &p, int problems, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3((unsigned)(problems * p.cs));
  cfg->blockDim = dim3(kC64Threads);
  cfg->dynamicSmemBytes = p.smem;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
}

}  // namespace

bool pcg_cluster64_plan(const ProblemInfo *prob, int num_problems, const int32_t *sblk_row, bool quad, int running,
                        Cluster64Plan *plan) {
  *plan = Cluster64Plan();
  int dev = 0, sms = 0, optin = 0;
  if (num_problems <= 0 || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  // per problem its cameras, the blocks of its rows of S (the diagonal ones
  // included), its longest row
  int n_max = 0, m_max = 1;
  long long w_max = 0;
  for (int p = 0; p < num_problems; ++p) {
    const int n = prob[p].cam_count, c0 = prob[p].cam_begin;
    if (n == 0) continue;
    n_max = std::max(n_max, n);
    w_max = std::max(w_max, (long long)(sblk_row[c0 + n] - sblk_row[c0]) + n);
    for (int c = c0; c < c0 + n; ++c) m_max = std::max(m_max, (int)(sblk_row[c + 1] - sblk_row[c]) + 1);
  }
  if (n_max <= 0 || n_max > kC64MaxCams || m_max > kC64MaxCams + 1) return false;
  const int nblk = (n_max + kPcgBlockCams - 1) / kPcgBlockCams;
  int nlev = 0;
  while ((1 << nlev) < m_max) ++nlev;
  // the cluster size and the rows per thread with the shortest estimated
  // iteration of the largest problem, in clocks: its product (FP64 warp
  // instructions on the busiest sub-partition), its tree, and the rest of
  // the chain (two cluster barriers and their exchanges when cs > 1), times
  // the waves of the launch
  double best = 1e300;
  for (int cs = 1; cs <= kC64MaxCS; cs *= 2)
    for (int R : {0, 1, 3, 9}) {
      const int rows = std::max(R, 1), U = 9 / rows;
      const long long pairs = (U * w_max + cs - 1) / cs + m_max;  // a run ends within one unit of its bound
      const int own = (nblk + cs - 1) / cs;
      if (pairs > 65535 || own > kC64Own) continue;
      const C64Layout l = c64_layout(R, n_max, own, (int)pairs);
      if (l.total + 4096 > (size_t)optin) continue;
      const double per_sm = std::max(1.0, std::floor((double)(228 * 1024) / (double)(l.total + 4096)));
      const double waves = std::max(1.0, std::ceil((double)running * cs / (sms * per_sm)));
      // CTAs that share an SM share its FP64 pipe
      const double share = std::min(per_sm, std::max(1.0, (double)running * cs / sms));
      double chain;
      if (R == 0) {
        const double m = (double)w_max / n_max, fit = std::max(1.0, std::floor(32.0 / m)), runs = std::ceil(m / 32.0);
        const double passes = std::ceil(9.0 * n_max / cs / fit) * runs, busy = std::ceil(passes / 4.0);
        chain = 76.0 * busy * share * (9.0 + std::ceil(std::log2(std::min(m, 32.0)))) + 200.0;
      } else {
        const double busy = std::ceil(std::ceil((double)pairs / 32.0) / 4.0);
        chain = 76.0 * 9.0 * R * busy * share + 300.0;
        for (int l2 = 0; l2 < nlev; ++l2)
          chain += 110.0 + 76.0 * R * std::ceil((double)pairs / (double)(2 << l2) / 128.0);
      }
      const double est = (chain + (cs == 1 ? 5500.0 : R == 0 ? 6500.0 : 8000.0)) * waves;
      if (est < best) {
        best = est;
        plan->cs = cs, plan->R = R, plan->n_max = n_max, plan->own_max = own, plan->pairs_max = (int)pairs;
        plan->smem = l.total, plan->clocks = est;
      }
    }
  // a single problem whose product keeps the cluster's 16 SMs busy for longer
  // goes to the grid form.  An iteration here and there, at the estimate in
  // thousands of clocks: 9.7 (39 cameras of a window) 5.5 and 6.2 us, 11.0 (24
  // cameras of a ring) 5.5 and 5.9, 11.6 (60 of a window) 6.7 and 6.5, 12.0
  // (32 of a ring) 6.6 and 6.2, 15.9 (75 of a walk) 8.9 and 6.9
  if (plan->cs == 0 || (num_problems == 1 && plan->clocks > kC64GridClocks)) {
    *plan = Cluster64Plan();
    return false;
  }
  plan->quad = quad;
  const void *f = (const void *)c64_kernel(plan->R, quad);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  c64_config(*plan, 1, &cfg, attr);
  int clusters = 0;
  if (raise_smem_limit(f, plan->smem) != cudaSuccess ||
      (plan->cs > 8 && cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    *plan = Cluster64Plan();
    return false;
  }
  return true;
}

cudaError_t launch_pcg_cluster64(const DeviceBatch &b, const Cluster64Plan &plan, cudaStream_t s) {
  if (b.num_problems == 0) return cudaSuccess;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  c64_config(plan, b.num_problems, &cfg, attr);
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, c64_kernel(plan.R, plan.quad), b, plan.cs, plan.n_max, plan.own_max, plan.pairs_max,
                            plan.above, plan.upto);
}

}  // namespace gba
