// k_pcg_grid.cu — the whole PCG of one problem in one launch spread over the
// whole GPU (FP64 form, explicit Schur complement), for problems whose rows
// of S do not fit a cluster (k_pcg_cluster64.cu) or keep it too busy.
//
// In the FP64 form a PCG iteration is a product with the 9x9 blocks of S
// (0.6 M FMAs on 250 cameras of a walk, about 1 us of the FP64 pipes of all
// SMs) between two problem-wide reductions; GB300 issues a dependent FP64
// instruction every 64 clocks, so the rest is the chain of the reductions
// and the exchanges between SMs through L2 (about 0.4 us a trip each way).
// One CTA per SM runs every iteration:
//   A. q = S p for the rows the CTA owns (runs of about equal numbers of row
//      blocks): p at the columns the rows touch and the rows of S in shared
//      memory, a thread per (row, block) pair (a nine-column FMA chain), each
//      row's block dots summed by the pairwise tree; q_i, and p_i q_i summed
//      over the row pairs (0,1) (2,3) (4,5) (6,7) of a camera (the first
//      level of sum9_tree; row 8 alone), are published;
//   B. the CTAs that own a chunk of 32 cameras: each camera's p.q from its
//      five values, the chunk's sum, published; every CTA: the chunks' sum (a
//      tree), alpha; for the camera blocks (8 cameras) the CTA owns: x, r,
//      z = M r, each block's r.z, r.r (and x.(v + r) when the stopping test
//      reads it), published with z;
//   C. every CTA: the sums over the blocks, the stopping test and beta in
//      warp 0, while the other warps fetch z of the touched columns;
//      p = z + beta p there.
// A published value is a 16-byte slot, the double and a tag of the launch
// and the iteration, written and read as one 128-bit access: a reader polls
// the slot itself until the tag is the one it waits for.  So an exchange
// costs the store's way to L2 and one read, no barrier, no fence and no
// second read; the slots alternate between two sets by iteration parity, and
// a set is only written again after every reader of its values has published
// what depends on them.  A CTA that owns nothing to publish therefore leaves
// (a row pair can cost more than a CTA's share: 20 of the 150 CTAs of a
// 30-camera walk own no unit, block or chunk).  One exchange from every CTA
// to every CTA would be 152 x 152 readers of the same lines (5 us, measured),
// so the p.q goes in two hops, over the CTAs that sum a chunk of 32 cameras,
// and what every CTA reads is published in kGridCopies copies.  A hop costs
// 0.4-1.3 us, most of it the lines' way between the SMs and the two dies' L2.
// Measured per PCG iteration, against two grid-wide counter barriers with the
// values read after them (which the values' copies and one read more replace):
// 75 cameras of a walk 8.1 -> 6.7 us, 120 8.5 -> 7.1, 170 8.9 -> 7.5, 250
// 9.9 -> 8.0.
// Left out, measured no faster: the CTAs that update camera blocks summing all
// chunks themselves (75 cameras 6.75 us as now, 250 8.4 against 8.2); slower:
// two warps or one pipelined warp polling a slot in turns (250 cameras 8.9 and
// 10.7 us), no copies, slots 128 bytes apart.
// Every CTA takes the same decisions from the same values.  The arithmetic
// is the two-kernel FP64 PCG's, operation for operation (the fixed trees of
// kernels.cuh, k_schur.cu's product and the camera kernel's reductions), so
// both forms give the same bits, and no result depends on how many CTAs took
// part.
//
// Participation.  The CTAs that start register on a counter; the first one
// closes the registration once every CTA of the launch has registered, or
// after kRegisterNs (another stream's kernels may hold SMs), and the work is
// split over the P CTAs that registered; a CTA that arrives after the
// closing leaves at once.  So every CTA waits only for CTAs that are running,
// whatever else the GPU is doing.  Every wait is bounded (kWaitNs, about a
// second): a CTA whose wait runs out raises the abort word, which ends every
// other CTA's waits; the problem's solve then ends with GBA_ERR_TIMEOUT in
// the status word and the LM loop stops.  The control words are zeroed, and
// the launch's tag counted up, by the camera Schur kernel K3b before each
// launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "kernels.h"

namespace gba {

namespace {

constexpr int kGThreads = kPcgGridThreads;
constexpr int kGWarps = kGThreads / 32;
constexpr int kGRows = 64;      // rows of one pass of the product (tables in shared memory)
constexpr int kGSteps = 12;     // steps of the pairwise tree, two levels each (rows of up to 2^24 blocks)
constexpr int kGBlkSlot = 96;   // threads per camera block in the update (3 warps)
constexpr int kGBlksPerRound = kGThreads / kGBlkSlot;
constexpr int kGMaxCams = 8192;  // cameras of the touched-column bitmap
static_assert(kGBlksPerRound >= 1 && kGThreads % 32 == 0 && kGWarps >= 4, "whole warps, at least one slot");
static_assert(kGBlkSlot % 32 == 0, "block slots of whole warps");
static_assert(9 * kPcgBlockCams <= kGBlkSlot, "a camera block's coordinates fit its slot");

constexpr unsigned long long kClosed = 1ull << 63;
constexpr unsigned long long kCountMask = 0xffffffffull;
constexpr unsigned long long kRegisterNs = 30000ull;    // stragglers of the launch, at most
constexpr unsigned long long kWaitNs = 1000000000ull;   // any other wait, at most

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Publishes a value: the slot's 16 bytes as one access.
__device__ __forceinline__ void slot_put(GridSlot *p, double v, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 r;\n\tmov.b128 r, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], r;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ unsigned long long slot_get(const GridSlot *p, double &v) {
  long long a;
  unsigned long long b;
  asm volatile("{\n\t.reg .b128 r;\n\tld.relaxed.gpu.global.b128 r, [%2];\n\tmov.b128 {%0, %1}, r;\n\t}"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
  v = __longlong_as_double(a);
  return b;
}

// Raises the abort word (first one wins) and records the timeout.
__device__ void grid_abort(const DeviceBatch &B) {
  if (atomicExch(B.grid_ctl + kGridAbort, 1u) == 0u)
    atomicExch(reinterpret_cast<unsigned *>(B.status), (unsigned)GBA_ERR_TIMEOUT);
}

// Waits until the N slots of every lane with `need` carry `tag` and returns
// their values; on a wait that ran out or was aborted sets the threads' *fail
// (the CTA's next checking barrier collects it).  Call from a whole warp: the lanes
// leave the loop together (lanes that left one by one would run on apart, an
// FP64 instruction issued for each).
template <int N>
__device__ __forceinline__ void slots_wait(const DeviceBatch &B, const GridSlot *const (&p)[N], unsigned long long tag,
                                           bool need, double (&v)[N], int *fail) {
  unsigned n = 0;
  unsigned long long t0 = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = 0.0;
  for (;;) {
    bool ok = true;
    if (need) {
#pragma unroll
      for (int j = 0; j < N; ++j) ok = (slot_get(p[j], v[j]) == tag) && ok;
    }
    if (__all_sync(0xffffffffu, ok)) return;
    if ((++n & 63u) == 0u) {
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > kWaitNs) grid_abort(B);
      if (__any_sync(0xffffffffu, ld_acquire_u32(B.grid_ctl + kGridAbort) != 0u)) {
        *fail = 1;
        return;
      }
    }
  }
}
__device__ __forceinline__ double slot_wait(const DeviceBatch &B, const GridSlot *p, unsigned long long tag, bool need,
                                            int *fail) {
  const GridSlot *const a[1] = {p};
  double v[1];
  slots_wait<1>(B, a, tag, need, v, fail);
  return v[0];
}

// Dynamic shared memory: the rows of the block-Jacobi inverse of the
// update's coordinates (one row per thread), the cameras' p.q chunk sums; per
// touched column its camera, the direction and z there; for the product's
// pass (at most kGRows rows, cap_pairs (row, block) pairs): each pair's row
// of S (when cached), dot and column, each row's first pair, the tree's steps.
struct GridSmem {
  size_t mrow, chs, clist, p, zc, sval, pd, pcol, ldst, roff, total;
};
__host__ __device__ inline size_t grid_align(size_t x) { return (x + 15) & ~size_t(15); }
__host__ __device__ inline GridSmem grid_smem(int n, int cap_cols, int cap_pairs) {
  GridSmem l;
  size_t o = 0;
  l.mrow = o, o = grid_align(o + 8 * 9 * (size_t)kGThreads);
  l.chs = o, o = grid_align(o + 8 * (size_t)((n + 31) / 32 + 1));
  l.clist = o, o = grid_align(o + 2 * (size_t)cap_cols);
  l.p = o, o = grid_align(o + 8 * 9 * (size_t)cap_cols);
  l.zc = o, o = grid_align(o + 8 * 9 * (size_t)cap_cols);
  l.sval = o, o = grid_align(o + 8 * 9 * (size_t)cap_pairs);
  l.pd = o, o = grid_align(o + 8 * (size_t)cap_pairs);
  l.pcol = o, o = grid_align(o + 4 * (size_t)cap_pairs);
  l.ldst = o, o = grid_align(o + 4 * (size_t)cap_pairs);
  l.roff = o, o = grid_align(o + 4 * (size_t)(kGRows + 1));
  l.total = o;
  return l;
}

// First row of unit u (5 per camera; kernels.h has the CTAs' shares).
__host__ __device__ inline int unit_row(int u) { return 9 * (u / 5) + 2 * (u % 5); }

// A tree step does two levels of the pairwise tree, s and 2 s: entry i (a
// multiple of 4 s with i + s < m) adds up to four sums, (i + i+s) +
// (i+2s + i+3s), those that exist.
__host__ __device__ __forceinline__ int step_entries(int m, int s) { return m > s ? (m - 1 - s) / (4 * s) + 1 : 0; }

}  // namespace

template <bool QUAD>
__global__ void __launch_bounds__(kGThreads, 1) k_pcg_grid(DeviceBatch B, int cap_cols, int cap_pairs) {
  extern __shared__ __align__(16) unsigned char g_smem[];
  __shared__ int s_ticket, s_P, s_ua, s_ub, s_stop, s_pass_end, s_npairs, s_nstep, s_good, s_ncol;
  __shared__ unsigned cmask[kGMaxCams / 32], cpre[kGMaxCams / 32];
  __shared__ int lbeg[kGSteps + 1];
  __shared__ double sc[3], s_inv_rz;
  __shared__ double rv[kGThreads];  // r_{k+1} of the update's coordinates, for M r
  __shared__ double red3[kGWarps][3];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned full = 0xffffffffu;
  LMState *L = B.lm;  // one problem
  // the same state in every CTA (written by the kernels before this one)
  if (!(L->active && L->pcg_active)) return;
  const ProblemInfo pi = B.prob[0];

  // ---- registration --------------------------------------------------------
  if (t == 0) {
    unsigned long long *reg = reinterpret_cast<unsigned long long *>(B.grid_ctl + kGridReg);
    const unsigned long long old = atomicAdd(reg, 1ull);
    int ticket = -1, P = 0;
    if (!(old & kClosed)) {
      ticket = (int)(old & kCountMask);
      if (ticket == 0) {
        const unsigned long long t0 = global_ns();
        while ((ld_acquire_u64(reg) & kCountMask) < gridDim.x && global_ns() - t0 < kRegisterNs) {
        }
        P = (int)(atomicOr(reg, kClosed) & kCountMask);
        st_release_u32(B.grid_ctl + kGridCount, (unsigned)P + 1u);
      } else {
        const unsigned long long t0 = global_ns();
        unsigned v;
        while ((v = ld_acquire_u32(B.grid_ctl + kGridCount)) == 0u) {
          if (global_ns() - t0 > kWaitNs) {
            grid_abort(B);
            break;
          }
        }
        if (v == 0u)
          ticket = -1;
        else
          P = (int)v - 1;
      }
    }
    s_ticket = ticket;
    s_P = P;
    s_ua = 0;
    s_ub = 0;
    s_ncol = 0;
  }
  for (int i = t; i < kGMaxCams / 32; i += kGThreads) cmask[i] = 0u;
  __syncthreads();
  const int w = s_ticket, P = s_P;
  if (w < 0) return;  // arrived after the closing (or the closing never came)

  // ---- ownership -------------------------------------------------------------
  // product: the problem's units in P runs of about equal cost
  const int n = pi.cam_count, c0 = pi.cam_begin;
  const int r0 = B.sblk_row[c0];
  {
    const long long wtot = (long long)(B.sblk_row[c0 + n] - r0) + n;
    const long long ta = grid_bound(w, P, wtot), tb = grid_bound(w + 1, P, wtot);
    int a = 0, b = 0;
    for (int c = t; c < n; c += kGThreads) {
      const long long before = (long long)(B.sblk_row[c0 + c] - r0) + c;
      const long long m = (long long)(B.sblk_row[c0 + c + 1] - B.sblk_row[c0 + c]) + 1;
      a += units5_below(ta, 9 * before, m);
      b += units5_below(tb, 9 * before, m);
    }
    if (a) atomicAdd(&s_ua, a);
    if (b) atomicAdd(&s_ub, b);
  }
  // update: camera blocks in P equal runs
  const int nblk = pi.cam_block_count;
  const int kb0 = grid_run(w, P, nblk), kb1 = grid_run(w + 1, P, nblk);
  // the chunks of 32 cameras whose p.q this CTA sums
  const int nch = (n + 31) / 32;
  const int ch0 = grid_run(w, P, nch), ch1 = grid_run(w + 1, P, nch);
  __syncthreads();
  const int ua = s_ua, nu = s_ub - ua;
  if (!grid_takes_part(nu, kb1 - kb0, ch1 - ch0)) return;  // (uniform; CTA 0 owns the first unit)
  const int ra = unit_row(ua), own_rows = nu > 0 ? unit_row(ua + nu) - ra : 0;  // rows of the problem (local)
  const double *vals = reinterpret_cast<const double *>(B.sblk_val);
  const double *Sii = reinterpret_cast<const double *>(B.cam_Sii);
  const GridSmem lay = grid_smem(n, cap_cols, cap_pairs);
  double *chs = reinterpret_cast<double *>(g_smem + lay.chs);
  unsigned short *clist = reinterpret_cast<unsigned short *>(g_smem + lay.clist);
  double *pc = reinterpret_cast<double *>(g_smem + lay.p);
  double *zc = reinterpret_cast<double *>(g_smem + lay.zc);
  double *sval = reinterpret_cast<double *>(g_smem + lay.sval);
  double *pd = reinterpret_cast<double *>(g_smem + lay.pd);
  int *pcol = reinterpret_cast<int *>(g_smem + lay.pcol);
  int *ldst = reinterpret_cast<int *>(g_smem + lay.ldst);
  int *roff = reinterpret_cast<int *>(g_smem + lay.roff);
  // the slots' two sets (by iteration parity): per row q, per coordinate z
  // and p, per unit p.q (by unit of the camera), and in kGridCopies copies
  // per chunk its p.q and per block its three sums
  const size_t n9 = 9 * (size_t)n;
  const size_t set = 3 * n9 + 5 * (size_t)n + kGridCopies * (3 * (size_t)nblk + (size_t)nch);
  GridSlot *const sl_q = B.grid_slots, *const sl_z = sl_q + n9, *const sl_p = sl_z + n9, *const sl_pq = sl_p + n9,
                  *const sl_c = sl_pq + 5 * (size_t)n, *const sl_b = sl_c + kGridCopies * (size_t)nch;
  const int copy = w % kGridCopies;  // the copy this CTA reads
  const unsigned long long launch_tag = (unsigned long long)B.grid_ctl[kGridLaunch] << 32;
  // (the failure test waits for a tag that nothing writes)
  const unsigned long long miss = B.opt.grid_wait_test ? 1ull << 31 : 0ull;

  auto row_m = [&](int rl) -> int {
    const int c = c0 + (ra + rl) / 9;
    return B.sblk_row[c + 1] - B.sblk_row[c] + 1;
  };
  // The product's pass over local rows [rl0, s_pass_end): whole units, at
  // most kGRows rows and cap_pairs (row, block) pairs; its tables: each row's
  // first pair (roff), each pair's column camera (pcol), the tree's steps
  // (ldst[lbeg[s] ..]: the first sum, and how many there are).
  auto build_pass = [&](int rl0) {
    if (t == 0) {
      int rl = rl0, np = 0, mx = 1;
      roff[0] = 0;
      while (rl < own_rows) {
        const int rows = (ra + rl) % 9 == 8 ? 1 : 2, m = row_m(rl);
        if (rl > rl0 && (np + rows * m > cap_pairs || rl + rows - rl0 > kGRows)) break;
        for (int r = 0; r < rows; ++r) np += m, ++rl, roff[rl - rl0] = np;
        mx = max(mx, m);
      }
      int ns = 0, o = 0;
      for (int s = 1; s < mx; s <<= 2, ++ns) {
        lbeg[ns] = o;
        for (int j = 0; j < rl - rl0; ++j) o += step_entries(roff[j + 1] - roff[j], s);
      }
      lbeg[ns] = o;
      s_pass_end = rl, s_npairs = np, s_nstep = ns;
    }
    __syncthreads();
    const int nr = s_pass_end - rl0, ns = s_nstep;
    for (int j = warp; j < nr; j += kGWarps) {
      const int c = (ra + rl0 + j) / 9, rr0 = B.sblk_row[c0 + c], m = roff[j + 1] - roff[j];
      for (int v = lane; v < m; v += 32) pcol[roff[j] + v] = v < m - 1 ? B.sblk_col[rr0 + v] - c0 : c;
    }
    for (int s2 = 0; s2 < ns; ++s2) {
      const int s = 1 << (2 * s2), base = lbeg[s2], cnt = lbeg[s2 + 1] - base;
      for (int kk = t; kk < cnt; kk += kGThreads) {
        int j = 0, acc = 0;
        for (;;) {
          const int a = step_entries(roff[j + 1] - roff[j], s);
          if (kk < acc + a) break;
          acc += a;
          ++j;
        }
        const int i = 4 * s * (kk - acc), m = roff[j + 1] - roff[j];
        ldst[base + kk] = (roff[j] + i) | (i + 3 * s < m ? 2 : i + 2 * s < m ? 1 : 0) << 28;
      }
    }
    __syncthreads();
  };
  bool one_pass = true, staged = false;
  int ncol = 0;
  if (own_rows > 0) {
    build_pass(0);
    one_pass = s_pass_end == own_rows;
    if (one_pass) {
      // the touched columns, in camera order, and the pairs' indexes among them
      const int np = s_npairs;
      for (int e = t; e < np; e += kGThreads) atomicOr(&cmask[pcol[e] >> 5], 1u << (pcol[e] & 31));
      __syncthreads();
      if (t == 0) {
        int o = 0;
        for (int i = 0; i < (n + 31) / 32; ++i) cpre[i] = o, o += __popc(cmask[i]);
        s_ncol = o;
      }
      __syncthreads();
      ncol = s_ncol;
      staged = ncol <= cap_cols;
      if (staged) {
        for (int c = t; c < n; c += kGThreads) {
          const unsigned bit = 1u << (c & 31);
          if (cmask[c >> 5] & bit) clist[cpre[c >> 5] + __popc(cmask[c >> 5] & (bit - 1u))] = (unsigned short)c;
        }
        for (int j = warp; j < own_rows; j += kGWarps) {
          const int c = (ra + j) / 9, q = ra + j - 9 * c, rr0 = B.sblk_row[c0 + c], m = roff[j + 1] - roff[j];
          for (int i = lane; i < 9 * m; i += 32) {
            const int v = i / 9, cc = i - 9 * v;
            sval[9 * roff[j] + i] = v < m - 1 ? vals[81 * (size_t)(rr0 + v) + 9 * q + cc] : Sii[81 * (size_t)(c0 + c) + 9 * q + cc];
          }
        }
        __syncthreads();
        for (int e = t; e < np; e += kGThreads) {
          const int c = pcol[e];
          pcol[e] = cpre[c >> 5] + __popc(cmask[c >> 5] & ((1u << (c & 31)) - 1u));
        }
        for (int e = t; e < 9 * ncol; e += kGThreads) pc[e] = B.pcg_z[9 * (size_t)(c0 + clist[e / 9]) + e % 9];  // p_0 = z_0
      }
    }
  }

  // the row that this thread publishes, when the CTA's rows are one pass: its
  // dot's and its own coordinates' addresses
  const double *w_d0 = pd, *w_d1 = pd, *w_p = pc;
  bool w_in = false, w_even = false, w_pair = false;
  int w_row = 0, w_unit = 0;
  // and its additions in the tree's steps (kGKeep of them at most, one entry
  // per thread in each; else from the tables)
  constexpr int kGKeep = 4;
  int w_tree[kGKeep];
  bool keep_tree = staged && s_nstep <= kGKeep;
  if (staged) {
    __syncthreads();
#pragma unroll
    for (int s2 = 0; s2 < kGKeep; ++s2) {
      w_tree[s2] = -1;
      if (s2 < s_nstep) {
        const int kk = lbeg[s2] + t;
        if (kk < lbeg[s2 + 1]) w_tree[s2] = ldst[kk];
        keep_tree = keep_tree && lbeg[s2 + 1] - lbeg[s2] <= kGThreads;
      }
    }
    w_in = t < own_rows;
    const int tr = min(t, own_rows - 1), cl = (ra + tr) / 9, q = ra + tr - 9 * cl;
    w_even = w_in && (q & 1) == 0, w_pair = w_even && q < 8;
    w_row = ra + tr, w_unit = (q >> 1) * n + cl;
    w_d0 = pd + roff[tr], w_d1 = pd + roff[w_pair ? tr + 1 : tr];
    w_p = pc + 9 * pcol[roff[tr + 1] - 1] + q;
  }

  const DeviceOptions &o = B.opt;
  double rz_k = L->rz, beta = L->beta, q0 = L->q0;
  double last_rr = L->rr, last_pq = L->pq;
  const double lim = o.pcg_tolerance * L->r0_norm;
  const long long lim2_bits = __double_as_longlong(lim * lim);
  int k = 0;
  // a wait of the thread's that ran out or was aborted: the two barriers that
  // check it carry it to every thread (a flag in shared memory could be set by
  // a warp past the check before the others have read it, and they would leave
  // that warp behind at its next barrier)
  int fail = 0;
  bool linear_ok = true, aborted = false;

  // the update's coordinate of this thread (coordinate m of a camera block
  // in the lanes of 3 warps); with at most kGBlksPerRound owned blocks its
  // state stays in registers, else in global memory
  const bool one_round = kb1 - kb0 <= kGBlksPerRound;
  const int u_slot = t / kGBlkSlot, u_m = t - kGBlkSlot * u_slot, u_q = u_m % 9;
  double ux = 0.0, ur = 0.0, uz = 0.0, uv = 0.0, up = 0.0;
  double *umrow = reinterpret_cast<double *>(g_smem + lay.mrow) + 9 * t;
  auto load_coordinate = [&](int blk, bool first) -> bool {  // of block blk; true in the threads that hold one
    const bool lead = u_slot < kGBlksPerRound && blk < kb1 && u_m < 9 * min(kPcgBlockCams, n - kPcgBlockCams * blk);
    if (lead) {
      const size_t i = 9 * (size_t)(c0 + kPcgBlockCams * blk) + u_m;
#pragma unroll
      for (int kk = 0; kk < 9; ++kk) umrow[kk] = B.cam_Minv[9 * i + kk];  // row u_q of the camera's block
      ux = B.pcg_x[i], ur = B.pcg_r[i], uz = B.pcg_z[i], uv = B.pcg_v[i];
      up = first ? 0.0 : B.pcg_p[i];
    }
    return lead;
  };
  bool u_lead = one_round && load_coordinate(kb0 + u_slot, true);
  __syncthreads();
  for (;;) {
    const unsigned long long tag = launch_tag | (unsigned)(k + 1);
    const unsigned long long wait_tag = tag ^ miss;
    const size_t so = (k & 1) ? set : 0;  // this iteration's slots
    // ---- the owned blocks' p_k, published for the CTAs that do not hold the
    // direction themselves (more rows or columns than the layout holds)
    if (one_round) {
      if (u_lead) {
        up = k == 0 ? uz : fma(beta, up, uz);
        slot_put(sl_p + so + kPcgBlockCams * 9 * (size_t)(kb0 + u_slot) + u_m, up, tag);
      }
    } else {
      for (int kb = kb0; kb < kb1; kb += kGBlksPerRound)
        if (load_coordinate(kb + u_slot, k == 0)) {
          const size_t i = kPcgBlockCams * 9 * (size_t)(kb + u_slot) + u_m;
          up = k == 0 ? uz : fma(beta, up, uz);
          B.pcg_p[9 * (size_t)c0 + i] = up;
          slot_put(sl_p + so + i, up, tag);
        }
    }
    // ---- A. q = S p_k for the owned rows, each unit's p_i q_i ---------------
    for (int rl0 = 0; rl0 < own_rows;) {
      if (!one_pass) build_pass(rl0);
      const int pend = one_pass ? own_rows : s_pass_end, np = s_npairs, ns = s_nstep;
      // the pairs' block dots (nine-column FMA chains)
      if (staged) {
        for (int e = t; e < np; e += kGThreads) {
          const double *row = sval + 9 * e, *pp = pc + 9 * pcol[e];
          double d = 0.0;
#pragma unroll
          for (int cc = 0; cc < 9; ++cc) d = fma(row[cc], pp[cc], d);
          pd[e] = d;
        }
      } else {
        for (int j = warp; j < pend - rl0; j += kGWarps) {
          const int rho = ra + rl0 + j, cl = rho / 9, q = rho - 9 * cl, rr0 = B.sblk_row[c0 + cl];
          const int m = roff[j + 1] - roff[j];
          for (int v0 = 0; v0 < m; v0 += 32) {
            const int v = min(v0 + lane, m - 1);
            const double *row = (v < m - 1 ? vals + 81 * (size_t)(rr0 + v) : Sii + 81 * (size_t)(c0 + cl)) + 9 * q;
            const GridSlot *ps = sl_p + so + 9 * (size_t)pcol[roff[j] + v];
            double d = 0.0;
            for (int cc = 0; cc < 9; ++cc) d = fma(row[cc], slot_wait(B, ps + cc, wait_tag, true, &fail), d);
            if (v0 + lane < m) pd[roff[j] + v] = d;
          }
        }
      }
      __syncthreads();
      // each row's pairwise tree, two levels a step
      auto step = [&](int e, int sp) {
        const int more = e >> 28;
        double *d = pd + (e & 0xfffffff);
        double x = d[0] + d[sp];
        if (more > 0) {
          double y = d[2 * sp];
          if (more > 1) y += d[3 * sp];
          x += y;
        }
        d[0] = x;
      };
      if (keep_tree) {
#pragma unroll
        for (int s2 = 0; s2 < kGKeep; ++s2)
          if (s2 < ns) {
            if (w_tree[s2] >= 0) step(w_tree[s2], 1 << (2 * s2));
            __syncthreads();
          }
      } else {
        for (int s2 = 0; s2 < ns; ++s2) {
          for (int kk = lbeg[s2] + t; kk < lbeg[s2 + 1]; kk += kGThreads) step(ldst[kk], 1 << (2 * s2));
          __syncthreads();
        }
      }
      // q_i per row and p_i q_i per unit (a thread each)
      if (staged) {
        if (32 * warp < own_rows) {
          const double qv = *w_d0, qv1 = *w_d1, p0 = w_p[0], p1 = w_pair ? w_p[1] : 0.0;
          if (w_in) slot_put(sl_q + so + w_row, qv, tag);
          const double y0 = __dmul_rn(p0, qv), y1 = __dadd_rn(y0, __dmul_rn(p1, qv1));
          if (w_even) slot_put(sl_pq + so + w_unit, w_pair ? y1 : y0, tag);
        }
      } else if (t < ((pend - rl0 + 31) & ~31)) {  // (whole warps)
        const bool in = t < pend - rl0;
        const int tr = min(t, pend - rl0 - 1);
        const int rho = ra + rl0 + tr, cl = rho / 9, q = rho - 9 * cl;
        const bool even = in && (q & 1) == 0, pair = even && q < 8;
        const double qv = pd[roff[tr]], qv1 = pair ? pd[roff[tr + 1]] : 0.0;
        if (in) slot_put(sl_q + so + rho, qv, tag);
        // p_k at the unit's own coordinates: the diagonal block's column
        const double p0 = slot_wait(B, sl_p + so + rho, wait_tag, even, &fail);
        const double p1 = slot_wait(B, sl_p + so + rho + (pair ? 1 : 0), wait_tag, pair, &fail);
        const double y0 = __dmul_rn(p0, qv), y1 = __dadd_rn(y0, __dmul_rn(p1, qv1));
        if (even) slot_put(sl_pq + so + (size_t)(q >> 1) * n + cl, pair ? y1 : y0, tag);
      }
      if (!one_pass) __syncthreads();  // pd and the pass tables are used again
      rl0 = pend;
    }
    // ---- B. the p.q of the CTA's chunks of 32 cameras, each camera's from
    // its five values (the rest of sum9_tree), then a butterfly; published.
    // The chunks from the last warp down: the first warps hold the update -----
    for (int j = ch0 + kGWarps - 1 - warp; j < ch1; j += kGWarps) {
      const int c = 32 * j + lane;
      const GridSlot *const pq0 = sl_pq + so + min(c, n - 1);
      const GridSlot *const a[5] = {pq0, pq0 + n, pq0 + 2 * (size_t)n, pq0 + 3 * (size_t)n, pq0 + 4 * (size_t)n};
      double y[5];
      slots_wait<5>(B, a, wait_tag, c < n, y, &fail);
      double x = ((y[0] + y[1]) + (y[2] + y[3])) + y[4];  // (0 beyond the problem's cameras)
      x = warp_sum(x);
      if (lane < kGridCopies) slot_put(sl_c + so + (size_t)lane * nch + j, x, tag);
    }
    // the owned coordinates' q; every CTA: the chunks' sum (the pairwise
    // tree: cta_chunked_sum's order), alpha; the update
    double qv = 0.0;
    if (one_round && __any_sync(full, u_lead))
      qv = slot_wait(B, sl_q + so + (u_lead ? kPcgBlockCams * 9 * (size_t)(kb0 + u_slot) + u_m : 0), wait_tag, u_lead, &fail);
    if (nch > 32) {
      for (int j0 = 32 * warp; j0 < nch; j0 += kGThreads) {
        const int j = min(j0 + lane, nch - 1);
        chs[j] = slot_wait(B, sl_c + so + (size_t)copy * nch + j, wait_tag, true, &fail);
      }
      __syncthreads();
      cta_pairwise_tree(chs, nch);
    }
    if (warp == 0) {
      double s2;
      if (nch <= 32) {  // the tree by one warp's shuffles
        s2 = slot_wait(B, sl_c + so + (size_t)copy * nch + min(lane, nch - 1), wait_tag, lane < nch, &fail);
        for (int s = 1; s < nch; s <<= 1) {
          const double y = __shfl_down_sync(full, s2, s);
          s2 += (lane & (2 * s - 1)) == 0 && lane + s < nch ? y : 0.0;
        }
      } else {
        s2 = chs[0];
      }
      if (lane == 0) {
        const long long b2 = __double_as_longlong(s2);
        sc[0] = s2, sc[1] = rz_k * recip_nr(s2);
        s_good = b2 > 0 && b2 < 0x7ff0000000000000LL;  // positive and finite
      }
    } else if (t == kGThreads - 32) {
      s_inv_rz = recip_nr(rz_k);  // for beta, off the deciding warp's chain
    }
    if (__syncthreads_or(fail)) {
      aborted = true;
      break;
    }
    const double pq = sc[0], alpha = sc[1];
    if (s_good == 0) {  // S is not positive definite along p_k: the PCG ends with x_k
      if (k == 0) linear_ok = false;
      break;
    }
    for (int kb = kb0; kb < kb1; kb += kGBlksPerRound) {
      const int blk = kb + u_slot;
      const bool in = u_slot < kGBlksPerRound && blk < kb1;  // uniform over the slot's three warps
      const int coords = in ? 9 * min(kPcgBlockCams, n - kPcgBlockCams * blk) : 0;
      const size_t i = kPcgBlockCams * 9 * (size_t)blk + u_m;
      bool lead = u_lead;
      if (!one_round) {
        lead = load_coordinate(blk, false);
        qv = slot_wait(B, sl_q + so + (lead ? i : 0), wait_tag, lead, &fail);
      }
      if (lead) {
        ur = fma(-alpha, qv, ur);
        rv[t] = ur;
      }
      __syncthreads();
      if (in && 32 * (warp - 3 * u_slot) < coords) {
        double rz = 0.0, rr = 0.0, qx = 0.0;
        if (lead) {
          double zz = 0;
#pragma unroll
          for (int kk = 0; kk < 9; ++kk) zz += umrow[kk] * rv[t - u_q + kk];
          uz = zz;
          slot_put(sl_z + so + i, uz, tag);
          rz = ur * uz, rr = ur * ur;
        }
        if (QUAD) {
          if (lead) {
            ux = fma(alpha, up, ux);
            qx = ux * (uv + ur);
          }
          warp_sum3(rz, rr, qx);
          if (lane == 0) red3[warp][0] = rz, red3[warp][1] = rr, red3[warp][2] = qx;
        } else {
          // both butterflies at once: lanes 0-15 end with r.z, 16-31 with r.r
          const bool lo = lane < 16;
          double v = (lo ? rz : rr) + __shfl_xor_sync(full, lo ? rr : rz, 16);
          v += __shfl_xor_sync(full, v, 8);
          v += __shfl_xor_sync(full, v, 4);
          v += __shfl_xor_sync(full, v, 2);
          v += __shfl_xor_sync(full, v, 1);
          if ((lane & 15) == 0) red3[warp][lane >> 4] = v;
        }
      }
      __syncthreads();
      // the block's sums, its warps in order (a warp without coordinates adds nothing)
      if (in && warp == 3 * u_slot) {
        constexpr int kSums = QUAD ? 3 : 2;
        const int u = lane % kSums, cp = lane / kSums;
        double b = red3[3 * u_slot][u];
        if (coords > 32) b += red3[3 * u_slot + 1][u];
        if (coords > 64) b += red3[3 * u_slot + 2][u];
        if (cp < kGridCopies) slot_put(sl_b + so + (size_t)(3 * cp + u) * nblk + blk, b, tag);
      }
      if (lead && !QUAD) ux = fma(alpha, up, ux);
      if (!one_round) {
        if (lead) {
          const size_t g = 9 * (size_t)c0 + i;
          B.pcg_x[g] = ux, B.pcg_r[g] = ur, B.pcg_z[g] = uz;
        }
        __syncthreads();  // rv and red3 are used again
      }
    }
    // ---- C. the stopping test on (x_{k+1}, r_{k+1}) and beta_{k+1} in warp 0,
    // from the blocks' values (the camera kernel's order), while the other
    // warps fetch z_{k+1} of the touched columns --------------------------------
    if (warp == 0) {
      double a = 0.0, b = 0.0, x = 0.0;
      for (int b0 = 0; b0 < nblk; b0 += 32) {
        const int bb = b0 + lane;
        const GridSlot *const p3 = sl_b + so + 3 * (size_t)copy * nblk + min(bb, nblk - 1);
        constexpr int N = QUAD ? 3 : 2;
        const GridSlot *s3[3] = {p3, p3 + nblk, p3 + 2 * (size_t)nblk};
        const GridSlot *const(&sN)[N] = *reinterpret_cast<const GridSlot *const(*)[N]>(&s3);
        double y[N];
        slots_wait<N>(B, sN, wait_tag, bb < nblk, y, &fail);
        if (b0 == 0)
          a = y[0], b = y[1], x = QUAD ? y[N - 1] : 0.0;
        else if (bb < nblk)
          a += y[0], b += y[1], x += QUAD ? y[N - 1] : 0.0;
      }
      // the blocks' owners published z before their sums: the other warps may
      // read it now (polling it from the start would slow the sums' way)
      asm volatile("bar.arrive 1, %0;" ::"n"(kGThreads) : "memory");
      const bool lo = lane < 16;
      double v = (lo ? a : b) + __shfl_xor_sync(full, lo ? b : a, 16);
      for (int s = nblk > 8 ? 8 : nblk > 4 ? 4 : nblk > 2 ? 2 : nblk > 1 ? 1 : 0; s > 0; s >>= 1)
        v += __shfl_xor_sync(full, v, s);  // (a level that would only add zeros is left out)
      const double rz1 = __shfl_sync(full, v, 0), rr1 = __shfl_sync(full, v, 16);
      const int k1 = k + 1;
      bool stop = false;
      if (QUAD) {
        const double qk = -warp_sum(x);  // Q(x) = x'Sx - 2 v'x = -x.(v + r)
        const double lhs = k1 * (qk - q0), rhs = o.eta * qk;
        const bool below = qk > 0.0 ? lhs < rhs : (qk < 0.0 ? lhs > rhs : q0 > 0.0);
        if (below && k1 >= o.min_pcg_iterations) stop = true;
        q0 = qk;
      } else if (__double_as_longlong(rr1) <= lim2_bits && k1 >= o.min_pcg_iterations) {
        stop = true;  // rr1 <= lim^2 (neither negative; a NaN's bits are above every number's)
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
      asm volatile("bar.sync 1, %0;" ::"n"(kGThreads) : "memory");
      if (staged)
        for (int e0 = 32 * (warp - 1); e0 < 9 * ncol; e0 += kGThreads - 32) {
          const int e = min(e0 + lane, 9 * ncol - 1), cl = e / 9;
          zc[e] = slot_wait(B, sl_z + so + 9 * (size_t)clist[cl] + (e - 9 * cl), wait_tag, true, &fail);
        }
    }
    if (__syncthreads_or(fail)) {
      aborted = true;
      break;
    }
    beta = sc[0];
    rz_k = sc[1];
    last_rr = sc[2];
    last_pq = pq;
    ++k;
    if (s_stop != 0) break;
    // p_k = z_k + beta_k p_{k-1} at the touched columns
    if (staged)
      for (int e = t; e < 9 * ncol; e += kGThreads) pc[e] = fma(beta, pc[e], zc[e]);
    __syncthreads();  // the direction; sc and s_stop are written again in the next iteration
  }
  // the owned coordinates' x, r, z and the last direction, as the two-kernel
  // form leaves them
  if (!aborted && u_lead) {
    const size_t g = 9 * (size_t)(c0 + kPcgBlockCams * (kb0 + u_slot)) + u_m;
    B.pcg_x[g] = ux, B.pcg_r[g] = ur, B.pcg_z[g] = uz;
    if (k > 0) B.pcg_p[g] = up;
  }
  if (w == 0 && t == 0) {
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
    if (aborted) {
      // a wait ran out: the solve stops here with GBA_ERR_TIMEOUT
      L->linear_ok = 0;
      L->active = 0;
    }
  }
}

static const void *grid_kernel(bool quad) {
  return quad ? (const void *)k_pcg_grid<true> : (const void *)k_pcg_grid<false>;
}

bool pcg_grid_plan(int num_problems, bool mixed, bool explicit_schur, int nc, const int32_t *sblk_row,
                   const int32_t *sblk_col, int ctas, bool quad, GridPlan *plan) {
  *plan = GridPlan();
  if (num_problems != 1 || mixed || !explicit_schur || nc <= 0 || nc > kGMaxCams || !sblk_row) return false;
  const void *kernel = grid_kernel(quad);
  int dev = 0, sms = 0, optin = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  // one CTA per SM at most, and no more CTAs than units
  const int grid = std::max(1, std::min(ctas > 0 ? std::min(ctas, sms) : sms, 5 * nc));
  // the kernel's split of the units (all CTAs registered): the most (row,
  // block) pairs and touched columns of a CTA, the longest row
  const long long wtot = (long long)(sblk_row[nc] - sblk_row[0]) + nc;
  auto m_of = [&](int c) { return (long long)(sblk_row[c + 1] - sblk_row[c]) + 1; };
  long long most_pairs = 0, m_max = 0;
  int most_cols = 0;
  for (int c = 0; c < nc; ++c) m_max = std::max(m_max, m_of(c));
  std::vector<int> seen(nc, -1);
  int c = 0, j = 0;  // the next unit: camera, unit of the camera
  long long before = 0;
  for (int r = 0; r < grid; ++r) {
    const long long tb = grid_bound(r + 1, grid, wtot);
    long long pairs = 0;
    int cols = 0;
    while (c < nc) {
      const long long m = m_of(c);
      if (9 * before + 2 * m * j >= tb) break;
      pairs += j == 4 ? m : 2 * m;
      if (seen[c] != r) cols += 1, seen[c] = r;
      for (int e = sblk_row[c]; e < sblk_row[c + 1]; ++e) {
        const int k = sblk_col[e];
        if (seen[k] != r) cols += 1, seen[k] = r;
      }
      if (++j == 5) j = 0, before += m, ++c;
    }
    most_pairs = std::max(most_pairs, pairs);
    most_cols = std::max(most_cols, cols);
  }
  const size_t static_bytes = fa.sharedSizeBytes + 1024;  // the kernel's static shared memory, with margin
  // room for a few CTAs fewer than launched; a pass holds one whole unit at
  // least.  The form pays off while every CTA keeps its rows of S in shared
  // memory for the launch; a complement too large for that is streamed from
  // memory on every PCG iteration, which the two-kernel product (a CTA per
  // camera row, the blocks loaded ahead of the wait) does better (1,800
  // cameras, 5.8M observations: 85 us per PCG iteration against 378 us here)
  const int cap_pairs = (int)std::max<long long>(2 * m_max, most_pairs + most_pairs / 4 + 64);
  const int cap_cols = std::min(nc, most_cols + most_cols / 4 + 16);
  if (cap_pairs >= 1 << 28) return false;
  const size_t smem = grid_smem(nc, cap_cols, cap_pairs).total;
  if (smem + static_bytes > (size_t)optin) return false;
  if (raise_smem_limit(kernel, smem) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kGThreads, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return false;
  }
  plan->grid = grid;
  plan->cap_cols = cap_cols;
  plan->cap_pairs = cap_pairs;
  plan->quad = quad;
  plan->smem = smem;
  return true;
}

cudaError_t launch_pcg_grid(const DeviceBatch &b, const GridPlan &plan, cudaStream_t s) {
  if (plan.grid <= 0) return cudaSuccess;
  if (plan.quad)
    k_pcg_grid<true><<<plan.grid, kGThreads, plan.smem, s>>>(b, plan.cap_cols, plan.cap_pairs);
  else
    k_pcg_grid<false><<<plan.grid, kGThreads, plan.smem, s>>>(b, plan.cap_cols, plan.cap_pairs);
  return cudaGetLastError();
}

}  // namespace gba
