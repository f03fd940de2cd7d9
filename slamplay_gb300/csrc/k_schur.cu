// k_schur.cu — the explicit Schur complement (gba_schur GBA_SCHUR_EXPLICIT).
//
// When the cameras' co-visibility is sparse, the reduced camera matrix
//   S = B + Dc^2 - W C^-1 W^T
// has few nonzero 9x9 camera-camera blocks: a 250-camera random walk has
// about 28 per camera, 2.3 MB in FP32, where the Jacobian the implicit
// mat-vec reads on every PCG iteration is 28 MB.  Then S is formed once per
// LM iteration (the points eliminated into camera-camera blocks, as Ceres'
// SPARSE_SCHUR and ITERATIVE_SCHUR with use_explicit_schur_complement do)
// and every PCG iteration multiplies by the blocks, which stay in L2.
//
// With L L^T = C_j^-1 (the point's 3x3 factor) and F_a = J_c^T J_p L of an
// observation a (9x3, formed by the point kernel K3a), the block of cameras
// (i, k) is -sum over the points both see of F_a F_b^T.
//
//  K3c k_schur_form (FP64), k_schur_form_mixed
//                     one CTA per block on or above the diagonal (k >= i):
//                     the F rows of 64 pairs per round staged in shared
//                     memory (the next round's loads in flight while this
//                     one is summed); the sum over the block's pairs, in a
//                     fixed order (three interleaved runs over the pairs'
//                     point order, combined in order; compensated FP32 in
//                     the mixed form), stored with its transpose as block
//                     (k, i).  The diagonal blocks B + Dc^2 - sum F_a F_a^T
//                     come from K3b; a camera that sees a point twice has a
//                     block (i, i) here for the cross terms.
//  K4a' k_schur_spmv  (FP64: k_schur_spmv64) one CTA per camera, or
//                     cameras in turn, one warp per row of its 9x9
//                     blocks, the lanes over the row's blocks (the last
//                     one the diagonal block): q = S p_k with p_k = z_k +
//                     beta_k p_{k-1} formed on the fly exactly as the
//                     implicit mat-vec forms it, and the camera's share of
//                     p.q for the camera kernel.  The blocks are fixed
//                     during the PCG, so their loads are issued before the
//                     wait on the preceding camera kernel.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"
#include "kernels.h"

namespace gba {

namespace {

constexpr int kFormPairs = 64;  // pairs per round
constexpr int kFormSub = 3;     // sub-lanes (interleaved runs) per block entry

__device__ __forceinline__ void pdl_wait_s() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents_s() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace

// ---------------------------------------------------------------------------
// K3c of the FP64 form, two CTAs a block (entries 0-40 and 41-80).  The FP64
// pipe bounds it: 243 FMAs a pair at one warp instruction per 64 clocks per
// sub-partition, dependent or not.  With four warps a CTA a lone block's
// three runs go at the chain's own speed (eight warps for all 81 entries on
// one SM take twice as long), and many blocks fill the GPU as before.  Every
// warp copies the F rows of eight of 32 pairs, asynchronously, the next 32's
// in flight while one is summed.  One CTA of eight warps a block, and now: 43
// and 27 us (rig window, blocks of up to 500 pairs), 53 and 41 (23 cameras),
// 520 and 430 (48 windows), 488 and 454 (250 cameras, 883,000 pairs; the
// FMAs alone 342).
constexpr int kForm64Warps = 4;
constexpr int kForm64Pairs = 32;
constexpr int kForm64Split = 41;  // entries of the first CTA
static_assert(kFormPairs == 2 * kForm64Pairs && kForm64Split * kFormSub <= 32 * kForm64Warps, "rounds and threads");

__global__ void __launch_bounds__(32 * kForm64Warps) k_schur_form(DeviceBatch B) {
  __shared__ __align__(16) double Fs[2][kForm64Pairs][2][kObsF];
  __shared__ double part[kFormSub][kForm64Split];
  constexpr int kWarpPairs = kForm64Pairs / kForm64Warps, kRowVecs = kObsF / 2;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int ub = blockIdx.x >> 1, blk = B.sblk_up[ub];
  const int p0 = B.sblk_pair[ub], p1 = B.sblk_pair[ub + 1];
  if (!B.lm[B.cam_problem[B.sblk_col[blk]]].active) return;  // uniform
  const double *F = reinterpret_cast<const double *>(B.obs_F);
  const int *pairs = reinterpret_cast<const int *>(B.spair);
  const int w0 = kWarpPairs * warp;
  // lane l < 16: the observation of the warp's pair l / 2, the row's (even) or the column's
  auto load_index = [&](int g) {
    return lane < 2 * kWarpPairs && g + w0 + (lane >> 1) < p1 ? pairs[2 * (size_t)(g + w0) + lane] : 0;
  };
  auto stage_rows = [&](int g, int st, int ob) {
    const int rows = 2 * (p1 - g - w0);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&Fs[st][w0][0][0]);
#pragma unroll
    for (int u = 0; u < 2 * kWarpPairs * kRowVecs / 32; ++u) {
      const int i = lane + 32 * u, row = i / kRowVecs, e = i - kRowVecs * row;
      const int o = __shfl_sync(0xffffffffu, ob, row);
      if (row < rows)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (uint32_t)i),
                     "l"(F + (size_t)kObsF * o + 2 * e)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // sub-lane `sub` of entry (i, k) sums the pairs sub, sub + kFormSub, ... of
  // every round of 64, in order: one FMA chain through the accumulator (three
  // FP64 operations a pair, not four)
  const int half = blockIdx.x & 1, tr = B.sblk_tr[blk];
  double *vals = reinterpret_cast<double *>(B.sblk_val);
  auto store = [&](int i, int k, double v) {
    vals[81 * (size_t)blk + 9 * i + k] = v;
    if (tr != blk) vals[81 * (size_t)tr + 9 * k + i] = v;
  };
  // a rig's poses have six parameters: its 36 entries by the first CTA, the
  // zeros (negated, as a sum would be) by the second
  const bool rig = B.opt.pinhole != 0;
  if (rig && half == 1) {
    if (t < 81 && (t / 9 >= 6 || t % 9 >= 6)) store(t / 9, t % 9, -0.0);
    return;
  }
  const int e0 = half * kForm64Split, cnt = rig ? 36 : min(kForm64Split, 81 - e0), wide = rig ? 6 : 9;
  const int sub = t / cnt, en = e0 + t - cnt * sub, ei = en / wide, ek = en - wide * ei;
  double acc = 0.0;
  stage_rows(p0, 0, load_index(p0));
  int ob = load_index(p0 + kForm64Pairs);
  int u = sub;  // the run's next pair of the round
  for (int g = p0, it = 0; g < p1; g += kForm64Pairs, ++it) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // these pairs have landed; every warp is done with the ones before
    stage_rows(g + kForm64Pairs, (it & 1) ^ 1, ob);
    ob = load_index(g + 2 * kForm64Pairs);
    const int base = kForm64Pairs * (it & 1), lim = base + min(kForm64Pairs, p1 - g);
    if (sub < kFormSub)
#pragma unroll 4
      for (; u < lim; u += kFormSub) {
        const double *fa = &Fs[it & 1][u - base][0][3 * ei], *fb = &Fs[it & 1][u - base][1][3 * ek];
        acc = fma(fa[2], fb[2], fma(fa[1], fb[1], fma(fa[0], fb[0], acc)));
      }
    if (it & 1) u = sub;
  }
  if (sub < kFormSub) part[sub][en - e0] = acc;
  __syncthreads();
  if (t < cnt) {
    double s = part[0][t];
#pragma unroll
    for (int j = 1; j < kFormSub; ++j) s += part[j][t];
    store((e0 + t) / wide, (e0 + t) % wide, -s);
  }
}

// K3c of the mixed form.  What bounded the form above there were its
// shared-memory loads, six per entry and pair: a lane here sums three entries
// of a column (four loads per entry and pair), three rows' thirds times three
// columns times the three interleaved runs on 27 lanes of three warps, with
// the same additions in the same order, the next step's rows loaded while
// one is added.  All four warps copy the F rows, 16 pairs of a round each,
// asynchronously, a round ahead.  Before and after, per launch: 882 and 535 us
// on 68,000 blocks of 107 pairs, 323 and 213 on 192 windows of 5-40 cameras,
// 122 and 87 on 250 cameras, 38 and 33 on one window of 8 cameras (blocks of
// up to 1,300 pairs: the chain of one block's steps bounds it).
constexpr int kTileWarps = 4;
constexpr int kTilePairs = 16;  // pairs of a round a warp copies
constexpr int kTileStages = 2;
static_assert(kFormPairs == kTileWarps * kTilePairs && kFormSub == 3, "stages of a round");
static_assert(kTilePairs * 2 == 32 && kObsF == 28, "a lane per row index, seven 16-byte copies a row");

// Entry e of block blk: its three runs combined in order, stored with the
// transpose.
__device__ __forceinline__ void store_mixed_entry(const DeviceBatch &B, const KahanF *part, int blk, int e) {
  KahanF s = part[e];
#pragma unroll
  for (int j = 1; j < kFormSub; ++j) s.merge(part[81 * j + e]);
  const float v = -s.rvalue();
  float *vals = reinterpret_cast<float *>(B.sblk_val);
  const int tr = B.sblk_tr[blk];
  vals[81 * (size_t)blk + e] = v;
  if (tr != blk) vals[81 * (size_t)tr + 9 * (e % 9) + e / 9] = v;
}

__global__ void __launch_bounds__(32 * kTileWarps) k_schur_form_mixed(DeviceBatch B) {
  __shared__ __align__(16) float Fs[kTileStages][kFormPairs][2][kObsF];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ub = blockIdx.x, blk = B.sblk_up[ub];
  const int p0 = B.sblk_pair[ub], p1 = B.sblk_pair[ub + 1];
  if (!B.lm[B.cam_problem[B.sblk_col[blk]]].active) return;  // uniform
  const float *F = reinterpret_cast<const float *>(B.obs_F);
  const int *pairs = reinterpret_cast<const int *>(B.spair);
  const int w0 = kTilePairs * warp;  // this warp's pairs of a round
  // lane l: the observation of the warp's pair l / 2, the row's (even) or the column's
  auto load_index = [&](int g) { return g + w0 + (lane >> 1) < p1 ? pairs[2 * (size_t)(g + w0) + lane] : 0; };
  // copies the rows of the warp's pairs of round g (none beyond p1)
  auto stage_rows = [&](int g, int st, int ob) {
    const int rows = 2 * (p1 - g - w0);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&Fs[st][w0][0][0]);
#pragma unroll
    for (int u = 0; u < 7; ++u) {
      const int i = lane + 32 * u, row = i / 7, e = i - 7 * row;
      const int o = __shfl_sync(0xffffffffu, ob, row);
      if (row < rows)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (uint32_t)i),
                     "l"(F + (size_t)kObsF * o + 4 * e)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int sub = lane / 9, tile = lane - 9 * sub, ti = tile / 3, kc = 3 * warp + tile - 3 * ti;
  const int last = min(sub, kFormSub - 1);  // (lanes 27-31 repeat a run's pairs and drop the result)
  const int busy = B.opt.pinhole ? 2 : 3;   // a rig's poses have six parameters: columns 6-8 stay zero
  KahanF acc[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) acc[e].init();
  struct Rows {
    float a[9], b[3];
  };
  auto load_rows = [&](int st, int r) {
    Rows f;
#pragma unroll
    for (int e = 0; e < 9; ++e) f.a[e] = Fs[st][r][0][9 * ti + e];
#pragma unroll
    for (int e = 0; e < 3; ++e) f.b[e] = Fs[st][r][1][3 * kc + e];
    return f;
  };
  auto add_rows = [&](const Rows &f) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      acc[i].add(f.a[3 * i] * f.b[0] + f.a[3 * i + 1] * f.b[1] + f.a[3 * i + 2] * f.b[2]);
  };
#pragma unroll
  for (int r = 0; r < kTileStages - 1; ++r) stage_rows(p0 + kFormPairs * r, r, load_index(p0 + kFormPairs * r));
  int ob = load_index(p0 + kFormPairs * (kTileStages - 1));
  for (int g = p0, st = 0; g < p1; g += kFormPairs) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kTileStages - 2) : "memory");
    __syncthreads();  // the round has landed; every warp is done with the one before
    stage_rows(g + kFormPairs * (kTileStages - 1), st == 0 ? kTileStages - 1 : st - 1, ob);
    ob = load_index(g + kFormPairs * kTileStages);
    if (warp < busy) {
      const int n = min(kFormPairs, p1 - g);
      int done = 0;
      if (n >= kFormSub) {
        Rows f = load_rows(st, last);
#pragma unroll 4
        for (done = kFormSub; done + kFormSub <= n; done += kFormSub) {
          const Rows nf = load_rows(st, done + last);
          add_rows(f);
          f = nf;
        }
        add_rows(f);
      }
      if (done + sub < n) add_rows(load_rows(st, done + sub));
    }
    st = st == kTileStages - 1 ? 0 : st + 1;
  }
  __syncthreads();  // the stages are reused
  KahanF *part = reinterpret_cast<KahanF *>(&Fs[0][0][0][0]);
  if (warp < 3 && sub < kFormSub)
#pragma unroll
    for (int i = 0; i < 3; ++i) part[81 * sub + 9 * (3 * ti + i) + kc] = acc[i];
  __syncthreads();
  if (threadIdx.x < 81) store_mixed_entry(B, part, blk, threadIdx.x);
}

// K3c of the mixed form when there are far more blocks than the GPU holds
// warps: a warp per block, a lane summing a 3x3 tile (two loads per entry and
// pair instead of four; 9 tiles times the three runs on 27 lanes), the warps
// independent of one another.  A long block is then one warp's chain, which
// many blocks hide and few do not.  The form above and this one, by blocks:
// 15,000 (100 windows) 269 and 316 us, 26,000 (1,800 cameras of a walk) 103
// and 82, 30,000 (200 windows) 445 and 431, 66,000 (1,800 cameras) 535 and
// 421, 100,000 (a walk) 307 and 197.  A round of 64 pairs comes 16 at
// a time, two of them ahead; the step of three pairs that crosses into the 16
// that just landed is done first, then the stage of the 16 before is free.
constexpr int kWarpFormBlocks = 24576;
constexpr int kWarpFormStages = 3;

__global__ void __launch_bounds__(32 * kTileWarps) k_schur_form_warp(DeviceBatch B) {
  __shared__ __align__(16) float Fs[kTileWarps][kWarpFormStages][kTilePairs][2][kObsF];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ub = blockIdx.x * kTileWarps + warp;
  if (ub >= B.nup) return;
  const int blk = B.sblk_up[ub];
  const int p0 = B.sblk_pair[ub], p1 = B.sblk_pair[ub + 1];
  if (!B.lm[B.cam_problem[B.sblk_col[blk]]].active) return;  // uniform over the warp
  const float *F = reinterpret_cast<const float *>(B.obs_F);
  const int *pairs = reinterpret_cast<const int *>(B.spair);
  // lane l: the observation of pair g + l / 2, the row's (even) or the column's
  auto load_index = [&](int g) { return g + (lane >> 1) < p1 ? pairs[2 * (size_t)g + lane] : 0; };
  auto stage_rows = [&](int g, int st, int ob) {  // the rows of pairs [g, g + 16), none beyond p1
    const int rows = 2 * (p1 - g);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&Fs[warp][st][0][0][0]);
#pragma unroll
    for (int u = 0; u < 7; ++u) {
      const int i = lane + 32 * u, row = i / 7, e = i - 7 * row;
      const int o = __shfl_sync(0xffffffffu, ob, row);
      if (row < rows)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (uint32_t)i),
                     "l"(F + (size_t)kObsF * o + 4 * e)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int sub = min(lane / 9, kFormSub), tile = lane - 9 * (lane / 9), ti = tile / 3, tk = tile - 3 * ti;
  const int last = min(sub, kFormSub - 1);  // (lanes 27-31 repeat a run's pairs and drop the result)
  KahanF acc[9];
#pragma unroll
  for (int e = 0; e < 9; ++e) acc[e].init();
  struct Rows {
    float a[9], b[9];
  };
  auto load_rows = [&](int st, int r) {  // of pair r of a stage
    Rows f;
    const float *fa = &Fs[warp][st][r][0][9 * ti], *fb = &Fs[warp][st][r][1][9 * tk];
#pragma unroll
    for (int e = 0; e < 9; ++e) f.a[e] = fa[e], f.b[e] = fb[e];
    return f;
  };
  auto add_rows = [&](const Rows &f) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k)
        acc[3 * i + k].add(f.a[3 * i] * f.b[3 * k] + f.a[3 * i + 1] * f.b[3 * k + 1] + f.a[3 * i + 2] * f.b[3 * k + 2]);
  };
  stage_rows(p0, 0, load_index(p0));
  stage_rows(p0 + kTilePairs, 1, load_index(p0 + kTilePairs));
  int ob = load_index(p0 + 2 * kTilePairs);
  int done = 0;  // pairs summed, from the start of the current 16 (negative: left over from the 16 before)
  int st = 0, prev = kWarpFormStages - 1;
  for (int g = p0, it = 0; g < p1; g += kTilePairs, ++it) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const int n = min(kTilePairs, p1 - g);
    if (done < 0 && done + kFormSub <= n) {
      const int r = done + last;
      add_rows(load_rows(r < 0 ? prev : st, r < 0 ? r + kTilePairs : r));
      done += kFormSub;
      __syncwarp();
    }
    // (a step still open here needs the stage of the 16 before, and nothing is left to copy)
    if (done >= 0) {
      stage_rows(g + 2 * kTilePairs, prev, ob);
      ob = load_index(g + 3 * kTilePairs);
    }
    if (done >= 0 && done + kFormSub <= n) {
      Rows f = load_rows(st, done + last);
#pragma unroll 2
      for (done += kFormSub; done + kFormSub <= n; done += kFormSub) {
        const Rows nf = load_rows(st, done + last);
        add_rows(f);
        f = nf;
      }
      add_rows(f);
    }
    if ((it & 3) == 3 || g + kTilePairs >= p1) {  // the round's last pairs
      const int r = done + sub;
      if (r < n) add_rows(load_rows(r < 0 ? prev : st, r < 0 ? r + kTilePairs : r));
      done = kTilePairs;
    }
    done -= kTilePairs;
    prev = st;
    st = st == kWarpFormStages - 1 ? 0 : st + 1;
    __syncwarp();
  }
  KahanF *part = reinterpret_cast<KahanF *>(&Fs[warp][0][0][0][0]);
  if (sub < kFormSub)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) part[81 * sub + 9 * (3 * ti + i) + 3 * tk + k] = acc[3 * i + k];
  __syncwarp();
  for (int e = lane; e < 81; e += 32) store_mixed_entry(B, part, blk, e);
}
static_assert(sizeof(KahanF) * 81 * kFormSub <= sizeof(float) * kWarpFormStages * kTilePairs * 2 * kObsF,
              "the runs fit the stages");
static_assert(kTilePairs % 3 == 1, "two pairs at most are left over from a stage");

void launch_schur_form(const DeviceBatch &b, bool mixed, cudaStream_t s) {
  if (!b.explicit_schur || b.nup == 0) return;
  if (mixed && b.nup >= kWarpFormBlocks)
    k_schur_form_warp<<<(b.nup + kTileWarps - 1) / kTileWarps, 32 * kTileWarps, 0, s>>>(b);
  else if (mixed)
    k_schur_form_mixed<<<b.nup, 32 * kTileWarps, 0, s>>>(b);
  else
    k_schur_form<<<2 * b.nup, 32 * kForm64Warps, 0, s>>>(b);
}

// ---------------------------------------------------------------------------
// K4a'
constexpr int kSpmvThreads = 9 * 32;
constexpr int kSpmvStage = 96;  // blocks of a camera staged at a time (at most)
constexpr int kSpmvCtas = 3;    // resident CTAs per SM
constexpr int kSpmvKeep = 8;    // cameras whose row sums a CTA keeps before it writes them

// Mixed form.  A lane that reads its block's row from memory touches a
// 128-byte line of its own with every load, and so do its reads of the
// direction: the L1's lines per load, not bytes, bounded the kernel.  So a
// camera's blocks, contiguous in memory, are copied into shared memory (16
// bytes a copy), the direction at their columns is formed once for the nine
// rows, and both are read from there, an odd stride between lanes (81 and 9
// words: no bank conflicts).  A camera needs a chain of loads (row, columns,
// direction, blocks), so a CTA takes every gridDim-th camera: the blocks of the next two cameras, the direction of the
// next and the columns of the one after are on their way while one is summed.
// The first two cameras' blocks are copied before the wait.  `cap` (a
// multiple of 32, at most kSpmvStage): blocks a stage holds; longer rows take
// rounds.  The rows' FP64 values are formed together for up to kSpmvKeep
// cameras (a warp for each row would queue on the FP64 pipes).  1,800 cameras
// of 74 blocks: 32.4 us reading from memory, 26.4 staged with a CTA per
// camera, 28.5 so pipelined with every warp reading the problem's state, 21.6
// now; instruction issue bounds it (some 600 a warp and camera).
__global__ void __launch_bounds__(kSpmvThreads, kSpmvCtas) k_schur_spmv(DeviceBatch B, int cap) {
  extern __shared__ __align__(16) float sv_smem[];  // two stages of [81 cap + 4] blocks, [9 cap] direction
  __shared__ float dg[81], own[kSpmvKeep][9];       // the diagonal block; the cameras' own direction
  __shared__ DF rows[kSpmvKeep][9];
  __shared__ double pqs[kSpmvKeep][9];
  __shared__ int kcam[kSpmvKeep];
  constexpr int kCols = 9 * kSpmvStage / kSpmvThreads;  // the direction's entries a thread forms
  const int t = threadIdx.x, q = t >> 5, lane = t & 31;
  float *sp = sv_smem + 2 * (81 * cap + 4);
  const uint32_t sv0 = (uint32_t)__cvta_generic_to_shared(sv_smem);
  struct Cam {
    int c, r0, nb, prob;
  };
  auto cam_at = [&](int i) {  // the CTA's i-th camera
    Cam m = {(int)(blockIdx.x + i * gridDim.x), 0, -1, -1};
    if (m.c < B.nc) {
      m.r0 = B.sblk_row[m.c];
      m.nb = B.sblk_row[m.c + 1] - m.r0;
      m.prob = B.cam_problem[m.c];
    }
    return m;
  };
  // The state of the cameras' problems: one thread reads it for the CTA (a
  // line that every warp of the GPU asks for is served by one slice of the
  // L2, a request a clock), past the L1, which would keep that of before the
  // wait.  Before the wait a PCG that is seen ended has ended, so an early
  // look only skips work.
  struct State {
    int live, k;
    float beta;
  };
  __shared__ State state[4];  // of the CTA's i-th camera: i mod 4
  State ns = {0, 0, 0.f};     // thread 0: the state read last, of problem nsp
  int nsp = -1;
  auto read_state = [&](const Cam &m) {
    if (t == 0 && m.prob != nsp) {
      nsp = m.prob;
      ns = State{0, 0, 0.f};
      if (nsp >= 0) {
        const LMState *L = B.lm + nsp;
        const int active = __ldcg(&L->active), pcg = __ldcg(&L->pcg_active), k = __ldcg(&L->pcg_iterations);
        const double beta = __ldcg(&L->beta);
        ns = State{active && pcg, k, (float)beta};
      }
    }
  };
  // blocks [v0, v0 + cap) of a camera's row, at their place in their 16 bytes
  auto stage = [&](const Cam &m, int st, int v0, bool live) {
    if (live) {
      const int n = min(cap, m.nb - v0), off = m.r0 & 3;
      const float *src = reinterpret_cast<const float *>(B.sblk_val) + 81 * (size_t)(m.r0 + v0) - off;
      const uint32_t dst = sv0 + 4u * (uint32_t)(st * (81 * cap + 4));
      for (int i = t; i < (n > 0 ? (off + 81 * n + 3) >> 2 : 0); i += kSpmvThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (uint32_t)i), "l"(src + 4 * (size_t)i)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the cameras whose direction this thread forms entries of (the row's
  // blocks in order, the diagonal block's, the camera itself, last)
  auto columns = [&](const Cam &m, int v0, int (&col)[kCols]) {
#pragma unroll
    for (int j = 0; j < kCols; ++j) {
      const int v = (t + j * kSpmvThreads) / 9;
      col[j] = -1;
      if (v < min(cap, m.nb + 1 - v0)) col[j] = v0 + v < m.nb ? B.sblk_col[m.r0 + v0 + v] : m.c;
    }
  };
  // p_k of a camera coordinate: the camera kernel's recurrence in FP32 on the
  // FP32 copies (as the implicit mat-vec)
  auto load_zp = [&](const int (&col)[kCols], float (&z)[kCols], float (&p)[kCols]) {
#pragma unroll
    for (int j = 0; j < kCols; ++j) {
      const int e = t + j * kSpmvThreads;
      z[j] = p[j] = 0.f;
      if (col[j] >= 0) {
        const size_t idx = 9 * (size_t)col[j] + (e - 9 * (e / 9));
        z[j] = B.pcg_zf[idx];
        p[j] = B.pcg_pf[idx];  // used when k > 0
      }
    }
  };
  const float *diag = reinterpret_cast<const float *>(B.cam_Sii);

  Cam m0 = cam_at(0), m1 = cam_at(1), m2 = cam_at(2);
  read_state(m0);
  if (t == 0) state[0] = ns;
  read_state(m1);
  if (t == 0) state[1] = ns;
  __syncthreads();
  stage(m0, 0, 0, state[0].live);
  stage(m1, 1, 0, state[1].live);
  int col1[kCols], col2[kCols];
  columns(m0, 0, col1);
  float d0 = m0.c < B.nc && t < 81 ? diag[81 * (size_t)m0.c + t] : 0.f;
  __syncthreads();  // the early states are read
  nsp = -1;
  pdl_wait_s();
  pdl_launch_dependents_s();
  float z0[kCols], p0[kCols], zo = 0.f, po = 0.f;
  load_zp(col1, z0, p0);
  if (m0.c < B.nc && t < 9) zo = B.pcg_zf[9 * (size_t)m0.c + t], po = B.pcg_pf[9 * (size_t)m0.c + t];
  columns(m1, 0, col1);
  read_state(m0);
  if (t == 0) state[0] = ns;
  read_state(m1);
  if (t == 0) state[1] = ns;
  read_state(m2);
  if (t == 0) state[2] = ns;
  __syncthreads();
  int kept = 0;
  // the kept cameras' rows and their shares of p.q
  auto write_kept = [&](int n) {
    __syncthreads();
    if (t < 9 * n) {
      const int i = t / 9, r = t - 9 * i;
      const double qv = df_value(rows[i][r]);
      B.pcg_q[9 * (size_t)kcam[i] + r] = qv;
      pqs[i][r] = (double)own[i][r] * qv;
    }
    __syncthreads();
    if (t < n) {
      double s = 0.0;
#pragma unroll
      for (int r = 0; r < 9; ++r) s += pqs[t][r];
      B.spmv_red[kcam[t]] = s;
    }
  };
  for (int i = 0; m0.c < B.nc; ++i) {
    if (t == 0 && i > 0) state[(i + 2) & 3] = ns;
    const int k = state[i & 3].k;
    const float beta = state[i & 3].beta;
    const bool live = state[i & 3].live;
    auto pdir = [&](float z, float p) { return k == 0 ? z : __fmaf_rn(beta, p, z); };
#pragma unroll
    for (int j = 0; j < kCols; ++j) {
      const int e = t + j * kSpmvThreads;
      if (e < 9 * cap) sp[e] = pdir(z0[j], p0[j]);
    }
    if (t < 81) dg[t] = d0;
    if (t < 9) own[kept][t] = pdir(zo, po);
    // the next camera's direction, the columns after it, the row after those
    if (m1.c < B.nc) {
      load_zp(col1, z0, p0);
      if (t < 9) zo = B.pcg_zf[9 * (size_t)m1.c + t], po = B.pcg_pf[9 * (size_t)m1.c + t];
      if (t < 81) d0 = diag[81 * (size_t)m1.c + t];
    }
    columns(m2, 0, col2);
    Cam m3 = cam_at(i + 3);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const int st = i & 1;
    if (live) {
      const float *sv = sv_smem + st * (81 * cap + 4) + (m0.r0 & 3);
      DF af = df_zero();  // the lane's blocks in order
      for (int v0 = 0;;) {
        const int n = min(cap, m0.nb + 1 - v0);
        for (int v = lane; v < n; v += 32) {
          const float *row = (v0 + v < m0.nb ? sv + 81 * v : dg) + 9 * q, *pp = sp + 9 * v;
          float s = 0.f;
#pragma unroll
          for (int cc = 0; cc < 9; ++cc) s += row[cc] * pp[cc];
          af = df_add(af, DF{s, 0.f});
        }
        if ((v0 += cap) > m0.nb) break;
        // a row longer than the stage: its next round, in line
        __syncthreads();
        stage(m0, st, v0, true);
        int col[kCols];
        float z[kCols], p[kCols];
        columns(m0, v0, col);
        load_zp(col, z, p);
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
          const int e = t + j * kSpmvThreads;
          if (e < 9 * cap) sp[e] = pdir(z[j], p[j]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
      }
      // the row's sum over the lanes (butterfly: a fixed order)
      af = df_warp_sum(af);
      if (lane == 0) rows[kept][q] = af;
      if (t == 0) kcam[kept] = m0.c;
    }
    __syncthreads();  // the stage is free
    stage(m2, st, 0, state[(i + 2) & 3].live);
    read_state(m3);
    if (live && ++kept == kSpmvKeep) {
      write_kept(kept);
      kept = 0;
    }
    m0 = m1, m1 = m2, m2 = m3;
#pragma unroll
    for (int j = 0; j < kCols; ++j) col1[j] = col2[j];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (kept > 0) write_kept(kept);
}

// K4a' of the FP64 form: one CTA per camera; the direction p_k = z_k +
// beta_k p_{k-1} at the columns of the camera's blocks formed once into
// shared memory (`stage`; else formed at each use, nine times per block),
// the block dots of its rows (nine-column FMA chains) into shared memory,
// `rpp` rows at a time, each row summed by the pairwise tree, then the
// camera's p.q (sum9_tree of its rows' p_i q_i): the grid PCG's arithmetic,
// so both forms agree bitwise.
__global__ void __launch_bounds__(kSpmvThreads) k_schur_spmv64(DeviceBatch B, int rpp, int stage) {
  extern __shared__ double sp_smem[];  // [m][9] staged direction (stage), then [rpp][m]
  __shared__ double pqs[9];
  const int c = blockIdx.x, t = threadIdx.x;
  const int prob = B.cam_problem[c];
  pdl_wait_s();
  pdl_launch_dependents_s();
  const LMState *L = B.lm + prob;
  if (!(L->active && L->pcg_active)) return;  // uniform over the CTA
  const int k = L->pcg_iterations;
  const double beta = L->beta;
  auto pdir = [&](size_t idx) -> double {
    const double z = B.pcg_z[idx];
    if (k == 0) return z;
    return fma(beta, B.pcg_p[idx], z);
  };
  const int r0 = B.sblk_row[c], nb = B.sblk_row[c + 1] - r0, m = nb + 1;
  const double *vals = reinterpret_cast<const double *>(B.sblk_val);
  const double *diag = reinterpret_cast<const double *>(B.cam_Sii) + 81 * (size_t)c;
  double *sp_p = sp_smem, *sp_d = sp_smem + (stage ? 9 * (size_t)m : 0);
  if (stage) {  // the diagonal block's column (the camera's own) last
    for (int e = t; e < 9 * m; e += kSpmvThreads) {
      const int v = e / 9, cc = e - 9 * v;
      sp_p[e] = pdir(9 * (size_t)(v < nb ? B.sblk_col[r0 + v] : c) + cc);
    }
    __syncthreads();
  }
  for (int q0 = 0; q0 < 9; q0 += rpp) {
    const int nr = min(rpp, 9 - q0);
    for (int e = t; e < nr * m; e += kSpmvThreads) {
      const int rr = e / m, v = e - rr * m;
      const double *row = (v < nb ? vals + 81 * (size_t)(r0 + v) : diag) + 9 * (q0 + rr);
      double d = 0.0;
      if (stage) {
        const double *pp = sp_p + 9 * v;
#pragma unroll
        for (int cc = 0; cc < 9; ++cc) d = fma(row[cc], pp[cc], d);
      } else {
        const int col = v < nb ? B.sblk_col[r0 + v] : c;
#pragma unroll
        for (int cc = 0; cc < 9; ++cc) d = fma(row[cc], pdir(9 * (size_t)col + cc), d);
      }
      sp_d[e] = d;
    }
    __syncthreads();
    for (int s = 1; s < m; s <<= 1) {
      const int na = tree_adds(m, s);
      for (int e = t; e < nr * na; e += kSpmvThreads) {
        const int rr = e / na, i = 2 * s * (e - rr * na);
        sp_d[rr * m + i] += sp_d[rr * m + i + s];
      }
      __syncthreads();
    }
    if (t < nr) {
      const int q = q0 + t;
      const size_t i = 9 * (size_t)c + q;
      const double qv = sp_d[t * m];
      B.pcg_q[i] = qv;
      pqs[q] = (stage ? sp_p[9 * nb + q] : pdir(i)) * qv;
    }
    __syncthreads();
  }
  if (t == 0) B.spmv_red[c] = sum9_tree(pqs);
}

// Rows per pass of k_schur_spmv64 and its shared memory, from the longest
// row (in blocks, the diagonal one included).
static int spmv64_rows(int m_max, size_t *smem, int *stage) {
  int optin = 48 * 1024, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t budget = (size_t)optin - 4096;
  const size_t mm = (size_t)std::max(m_max, 1);
  // the staged direction when it leaves room for one row's block dots
  *stage = 8 * 10 * mm <= budget ? 1 : 0;
  const size_t rows_budget = budget - (*stage ? 8 * 9 * mm : 0);
  int rpp = 9;
  while (rpp > 1 && 8 * (size_t)rpp * mm > rows_budget) --rpp;
  *smem = 8 * (size_t)rpp * mm + (*stage ? 8 * 9 * mm : 0);
  return rpp;
}

cudaError_t launch_schur_spmv(const DeviceBatch &b, bool mixed, cudaStream_t s, bool pdl) {
  if (b.nc == 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)b.nc);
  cfg.blockDim = dim3(kSpmvThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  if (mixed) {
    const int cap = std::min((b.sblk_max + 31) / 32 * 32, kSpmvStage);
    const size_t bytes = sizeof(float) * (2 * (81 * (size_t)cap + 4) + 9 * (size_t)cap);
    int sms = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = raise_smem_limit((const void *)k_schur_spmv, bytes);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3((unsigned)std::min(b.nc, kSpmvCtas * sms));
    cfg.dynamicSmemBytes = bytes;
    return cudaLaunchKernelEx(&cfg, k_schur_spmv, b, cap);
  }
  size_t smem = 0;
  int stage = 0;
  const int rpp = spmv64_rows(b.sblk_max, &smem, &stage);
  if (smem > 48 * 1024) {
    const cudaError_t e = raise_smem_limit((const void *)k_schur_spmv64, smem);
    if (e != cudaSuccess) return e;
  }
  cfg.dynamicSmemBytes = smem;
  return cudaLaunchKernelEx(&cfg, k_schur_spmv64, b, rpp, stage);
}

}  // namespace gba
