// k_pcg_cluster.cu — the whole PCG of a problem in one launch: one thread
// block cluster per problem (mixed form, explicit Schur complement).
//
// The two-kernel PCG (k_pcg.cu, k_schur.cu) pays two kernel boundaries per
// iteration, and a batch iterates until its slowest problem's PCG ends.
// Here a cluster of cs CTAs (cs <= 16, on cs SMs of one GPC) runs every
// iteration of one problem's PCG.  CTA `rank` owns a contiguous run of the
// problem's cameras and keeps x, r, v, q and its rows of S (when they fit)
// in shared memory; every CTA keeps p of the cameras that its rows touch and
// updates it with the same arithmetic, so the copies agree bitwise.  The
// direction is FP32 (the product's input) and the same FP32 values enter
// p.q and the update of x, so the curvature p.Sp and the recurrences refer
// to the direction the product used.  Per iteration:
//   1. q = S p for the owned rows (FP32 products and per-thread sums,
//      double-float across the threads of a row) and each owned camera's
//      p.q; cluster barrier
//   2. p.q over the problem's cameras, alpha; r and z = M r of the owned
//      cameras, each owned camera's r.z, r.r (and x.(v + r) when the stopping
//      test reads it); cluster barrier, x while it is on its way
//   3. the stopping test and beta from the cameras' values, p_{k+1} =
//      z_{k+1} + beta p_k for the touched cameras.
// What bounds an iteration is its chain: about 25 dependent double-float
// additions (some 60 clocks each, more where a warp adds several values, so
// the trees spread a group's sums over its lanes), the reads of S from
// shared memory, two cluster barriers and two read-backs (500 clocks each)
// when cs > 1.  Measured per PCG iteration, before the sums were spread and
// the direction limited to the touched cameras -> now: 250 cameras 8.2 ->
// 6.1 us, 23 cameras 5.0 -> 3.5 us, 7 cameras 2.0 -> 1.3 us.
// Each CTA stores its z and per-camera values into its own shared memory;
// after the cluster barrier (release/acquire) the others read them from
// there (distributed shared memory), one load per value.  The dot products
// are summed per camera (a fixed tree over its nine coordinates) and then
// over the problem's cameras (a fixed tree over a warp), so the result
// depends neither on the cluster size nor on the batch: a problem gets the
// same bits alone and in any batch.
// GB300 issues FP64 some 64 times slower than FP32 (and with a long
// latency), so the vectors and the PCG scalars are double-float (two
// floats, about 48 bits); the mixed form's matrix (S, M) is FP32, so this
// loses nothing FP64 vectors would keep.  Every CTA takes the same decisions
// from the same values, so all reach the same cluster barriers (the
// hardware's barrier.cluster arrive/wait; there are no spin-waits).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace gba {

namespace {

constexpr int kClSub = 8;  // lanes per (camera, row triplet) of the product

// Shared-memory layout (bytes), the same on the host and the device.
struct ClLayout {
  size_t zf, ph, mo, xh, xl, rh, rl, vh, vl, qh, ql, cpq, crr, cxv, owner, boff, scol, sval, total;
};
__host__ __device__ inline size_t cl_align(size_t x) { return (x + 15) & ~size_t(15); }
__host__ __device__ inline ClLayout cl_layout(int n_max, int own_max, int cache_blocks) {
  ClLayout l;
  size_t o = 0;
  const size_t nf = 4 * 9 * (size_t)n_max, of = 4 * 9 * (size_t)own_max;
  l.zf = o, o = cl_align(o + nf);
  l.ph = o, o = cl_align(o + 4 * 12 * (size_t)n_max);  // p, 12 floats per camera (three 16-byte loads)
  l.mo = o, o = cl_align(o + 4 * 81 * (size_t)own_max);
  l.xh = o, o = cl_align(o + of);
  l.xl = o, o = cl_align(o + of);
  l.rh = o, o = cl_align(o + of);
  l.rl = o, o = cl_align(o + of);
  l.vh = o, o = cl_align(o + of);
  l.vl = o, o = cl_align(o + of);
  l.qh = o, o = cl_align(o + of);
  l.ql = o, o = cl_align(o + of);
  // per camera, double-float: p.q; r.z and r.r; x.(v + r)
  l.cpq = o, o = cl_align(o + 8 * (size_t)n_max);
  l.crr = o, o = cl_align(o + 16 * (size_t)n_max);
  l.cxv = o, o = cl_align(o + 8 * (size_t)n_max);
  l.owner = o, o = cl_align(o + 4 * (size_t)n_max);    // per camera: the rank that owns it
  // the owned rows of S (cache_blocks > 0): per owned camera its first
  // block, per block its column camera (in the problem) and its 81 values
  l.boff = o, o = cl_align(o + (cache_blocks > 0 ? 4 * ((size_t)own_max + 1) : 0));
  l.scol = o, o = cl_align(o + 4 * (size_t)cache_blocks);
  // per block three row triplets (rows g, g + 3, g + 6) of 27 values + pad
  l.sval = o, o = cl_align(o + 4 * 84 * (size_t)cache_blocks);
  l.total = o;
  return l;
}

// Sum over the 16 lanes of a half-warp group (xor butterfly: a fixed tree,
// the same bits in every lane).
__device__ __forceinline__ DF df_group16_sum(DF v, unsigned mask) {
#pragma unroll
  for (int off = 1; off < 16; off <<= 1) {
    const DF w{__shfl_xor_sync(mask, v.hi, off), __shfl_xor_sync(mask, v.lo, off)};
    v = df_add(v, w);
  }
  return v;
}

// Sum of the problem's n per-camera values (staged in shared memory, value c
// at camv[stride c]; in one warp: lane l adds cameras l, l + 32, ... in
// order, then a butterfly, whose levels that would only add zeros are left
// out: adding zero changes no normalised pair); the total in lane 0.
__device__ __forceinline__ DF cam_total(const float2 *camv, int stride, int n) {
  const int lane = threadIdx.x & 31;
  DF s = df_zero();
  if (lane < n) {
    const float2 v = camv[stride * lane];
    s = DF{v.x, v.y};
  }
  for (int c = lane + 32; c < n; c += 32) {
    const float2 v = camv[stride * c];
    s = df_add(s, DF{v.x, v.y});
  }
  for (int o = n > 16 ? 16 : n > 8 ? 8 : n > 4 ? 4 : n > 2 ? 2 : n > 1 ? 1 : 0; o > 0; o >>= 1) {
    const DF w{__shfl_xor_sync(0xffffffffu, s.hi, o), __shfl_xor_sync(0xffffffffu, s.lo, o)};
    s = df_add(s, w);
  }
  return s;
}

// a / b in double-float: a float quotient, one correction step
__device__ __forceinline__ DF df_div(DF a, DF b) {
  const float q1 = __fdiv_rn(a.hi, b.hi);
  const DF r = df_add(a, df_neg(df_mul_f(b, q1)));
  const float q2 = __fdiv_rn(r.hi, b.hi);
  return df_fast_two_sum(q1, q2);
}
__device__ __forceinline__ bool df_le(DF a, DF b) { return a.hi < b.hi || (a.hi == b.hi && a.lo <= b.lo); }

// Shared memory of another CTA of the cluster.
template <typename T>
__device__ __forceinline__ T *peer(T *local, int rank) {
  return cg::this_cluster().map_shared_rank(local, rank);
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace

// QUAD: the quadratic-model stopping test, the only reader of x.(v + r).
template <bool QUAD>
__global__ void __launch_bounds__(kClThreads, 1) k_pcg_cluster(DeviceBatch B, int cs, int n_max, int own_max,
                                                            int cache_blocks, int above, int upto) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  const ClLayout lay = cl_layout(n_max, own_max, cache_blocks);
  float *zf = reinterpret_cast<float *>(cl_smem + lay.zf);
  float *ph = reinterpret_cast<float *>(cl_smem + lay.ph);
  float *Mo = reinterpret_cast<float *>(cl_smem + lay.mo);
  float *xh = reinterpret_cast<float *>(cl_smem + lay.xh);
  float *xl = reinterpret_cast<float *>(cl_smem + lay.xl);
  float *rh = reinterpret_cast<float *>(cl_smem + lay.rh);
  float *rl = reinterpret_cast<float *>(cl_smem + lay.rl);
  float *vh = reinterpret_cast<float *>(cl_smem + lay.vh);
  float *vl = reinterpret_cast<float *>(cl_smem + lay.vl);
  float *qh = reinterpret_cast<float *>(cl_smem + lay.qh);
  float *ql = reinterpret_cast<float *>(cl_smem + lay.ql);
  float2 *cpq = reinterpret_cast<float2 *>(cl_smem + lay.cpq);
  float4 *crr = reinterpret_cast<float4 *>(cl_smem + lay.crr);
  float2 *cxv = reinterpret_cast<float2 *>(cl_smem + lay.cxv);
  int *own_of = reinterpret_cast<int *>(cl_smem + lay.owner);
  int *boff = reinterpret_cast<int *>(cl_smem + lay.boff);
  int *scol = reinterpret_cast<int *>(cl_smem + lay.scol);
  float *sval = reinterpret_cast<float *>(cl_smem + lay.sval);
  __shared__ DF scf[4];
  __shared__ int s_lo, s_hi;

  const int rank = cs > 1 ? (int)cg::this_cluster().block_rank() : 0;
  // (the count of running PCGs that K3b left; the other shape takes this one)
  const int running = B.status[3];
  if (running <= above || running > upto) return;
  const int prob = B.prob_order[blockIdx.x / cs];  // the longest first: the short ones fill in behind
  const int t = threadIdx.x, T = blockDim.x;
  LMState *L = B.lm + prob;
  // uniform over the cluster: every CTA reads the same state before its
  // first barrier, and rank 0 changes it only after the last one
  if (!(L->active && L->pcg_active)) return;
  const ProblemInfo pi = B.prob[prob];
  const int n = pi.cam_count, c0 = pi.cam_begin;
  // the cameras split into cs runs of about equal blocks of S (the
  // product's work): CTA `rank` owns the cameras whose blocks before them
  // (with the diagonal ones) lie in [bound(rank), bound(rank + 1))
  // (bound(r) = ceil(r W / cs) <= before(c) exactly when r <= before(c) cs / W,
  // so camera c's owner is floor(before(c) cs / W))
  int own0 = 0, own_end = 0;
  {
    const int r0 = B.sblk_row[c0];
    const long long wtot = (long long)(B.sblk_row[c0 + n] - r0) + n;
    const long long ta = ((long long)rank * wtot + cs - 1) / cs, tb = ((long long)(rank + 1) * wtot + cs - 1) / cs;
    for (int cb = 0; cb < n; cb += T) {
      const int c = cb + t;
      const long long before = c < n ? (long long)(B.sblk_row[c0 + c] - r0) + c : wtot;
      if (c < n) own_of[c] = (int)(before * cs / wtot);
      own0 += __syncthreads_count(before < ta);
      own_end += __syncthreads_count(before < tb);
    }
  }
  const int own_n = own_end - own0;
  const int o9 = 9 * own_n, a9 = 9 * own0;  // a9: first owned coordinate in the problem
  const size_t g0 = 9 * (size_t)c0;                       // the problem's first coordinate (global)

  for (int i = t; i < o9; i += T) {
    const DF v = df_from_double(B.pcg_v[g0 + a9 + i]);
    const DF r = df_from_double(B.pcg_r[g0 + a9 + i]);
    xh[i] = 0.f, xl[i] = 0.f;
    rh[i] = r.hi, rl[i] = r.lo;
    vh[i] = v.hi, vl[i] = v.lo;
  }
  for (int i = t; i < 81 * own_n; i += T) Mo[i] = B.cam_Minvf[81 * (size_t)(c0 + own0) + i];
  const float *vals = reinterpret_cast<const float *>(B.sblk_val);
  const float *Sii = reinterpret_cast<const float *>(B.cam_Sii);
  const bool cached = cache_blocks > 0;
  if (cached) {
    // the owned rows of S, fixed during the PCG: off-diagonal blocks, then
    // the diagonal block, per owned camera
    if (t == 0) {
      int s = 0;
      for (int lc = 0; lc < own_n; ++lc) {
        boff[lc] = s;
        const int c = c0 + own0 + lc;
        s += B.sblk_row[c + 1] - B.sblk_row[c] + 1;
      }
      boff[own_n] = s;
    }
    __syncthreads();
    for (int lc = 0; lc < own_n; ++lc) {
      const int c = c0 + own0 + lc;
      const int r0 = B.sblk_row[c], nb = B.sblk_row[c + 1] - r0, b0 = boff[lc];
      for (int v = t; v <= nb; v += T) scol[b0 + v] = (v < nb ? B.sblk_col[r0 + v] : c) - c0;
      // triplet layout: block b, triplet g, entry j = row (g + 3 (j / 9)), column j % 9
      for (int e = t; e < 84 * (nb + 1); e += T) {
        const int v = e / 84, w = e - 84 * v, g = w / 28, j = w - 28 * g;
        float x = 0.f;
        if (j < 27) {
          const int el = 9 * (g + 3 * (j / 9)) + j % 9;
          x = v < nb ? vals[81 * (size_t)(r0 + v) + el] : Sii[81 * (size_t)c + el];
        }
        sval[84 * (size_t)(b0 + v) + w] = x;
      }
    }
  }
  // the cameras whose direction the CTA needs: the columns of the owned rows
  // (its own cameras among them)
  if (t == 0) s_lo = n, s_hi = -1;
  __syncthreads();
  if (own_n > 0) {
    int lo = own0, hi = own_end - 1;
    for (int e = B.sblk_row[c0 + own0] + t; e < B.sblk_row[c0 + own_end]; e += T) {
      const int c = B.sblk_col[e] - c0;
      lo = min(lo, c), hi = max(hi, c);
    }
    lo = __reduce_min_sync(0xffffffffu, lo), hi = __reduce_max_sync(0xffffffffu, hi);
    if ((t & 31) == 0) atomicMin(&s_lo, lo), atomicMax(&s_hi, hi);
  }
  __syncthreads();
  const int i_lo = 9 * s_lo, i_hi = 9 * (s_hi + 1);
  // the start (K3b): x = 0, r = v, z = M r, p_0 = z
  for (int i = i_lo + t; i < i_hi; i += T) {
    const float z = B.pcg_zf[g0 + i];
    zf[i] = z, ph[i + 3 * (i / 9)] = z;
  }
  const DeviceOptions &o = B.opt;
  // PCG scalars (double-float in every thread, the same values)
  DF rz = df_from_double(L->rz);
  double q0 = L->q0;
  const double lim = o.pcg_tolerance * L->r0_norm;
  const DF lim2 = df_from_double(lim * lim);
  int k = 0;
  bool linear_ok = true;
  DF last_pq = df_zero(), last_beta = df_zero(), last_rr = df_from_double(L->rr);
  const int lane = t % kClSub;
  // the lanes of a row group (kClSub consecutive lanes of a warp)
  const unsigned gmask = ((1u << kClSub) - 1u) << ((t & 31) & ~(kClSub - 1));
  // camera-coordinate mapping of the per-camera sums: a half-warp per camera
  const int hq = t & 15, hc = t >> 4;
  const int wc = hc & ~1;  // the warp's first camera: a warp without one does not take issue slots from the others
  const unsigned hmask = 0xffffu << (t & 16);
  __syncthreads();
  // the thread's first triplet of S stays in registers: reading S from
  // shared memory, seven 16-byte loads a triplet, bounds the product (the PCG
  // of an LM iteration, without and with: 379 and 363 us on 250 cameras, 563
  // and 549 on 192 windows; two triplets spill, 365 and 564)
  float sreg[27];
  int preg = -1;  // its column camera's p
  const int ws0 = t / kClSub;
  if (cached && ws0 < 3 * own_n) {
    const int lc = ws0 / 3, g = ws0 - 3 * lc, b = boff[lc] + lane;
    if (b < boff[lc + 1]) {
      preg = 12 * scol[b];
#pragma unroll
      for (int j = 0; j < 27; ++j) sreg[j] = sval[84 * b + 28 * g + j];
    }
  }
  for (;;) {
    // 1. q = S p_k for the owned rows: a thread takes rows g, g + 3, g + 6
    // of a camera (one load of p per block for three rows) for the blocks
    // lane, lane + kClSub, ... of the row (the last one the diagonal
    // block); FP32 sums per thread, double-float over the kClSub lanes
    for (int ws = t / kClSub; ws < 3 * own_n; ws += T / kClSub) {
      const int lc = ws / 3, g = ws - 3 * lc;
      const int c = c0 + own0 + lc;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f;
      if (cached) {
        const int b0 = boff[lc], nb1 = boff[lc + 1] - b0;
        int v = lane;
        if (ws == ws0) {
          v += kClSub;
          if (preg >= 0) {
            const float4 *p4 = reinterpret_cast<const float4 *>(ph + preg);
            float pv[12];
#pragma unroll
            for (int u = 0; u < 3; ++u) *reinterpret_cast<float4 *>(&pv[4 * u]) = p4[u];
#pragma unroll
            for (int cc = 0; cc < 9; ++cc) {
              a0 = __fmaf_rn(sreg[cc], pv[cc], a0);
              a1 = __fmaf_rn(sreg[9 + cc], pv[cc], a1);
              a2 = __fmaf_rn(sreg[18 + cc], pv[cc], a2);
            }
          }
        }
        for (; v < nb1; v += kClSub) {
          // the triplet's 27 values and the column camera's p: 16-byte loads
          const float4 *r4 = reinterpret_cast<const float4 *>(sval + 84 * (b0 + v) + 28 * g);
          const float4 *p4 = reinterpret_cast<const float4 *>(ph + 12 * scol[b0 + v]);
          float rv[28], pv[12];
#pragma unroll
          for (int u = 0; u < 7; ++u) *reinterpret_cast<float4 *>(&rv[4 * u]) = r4[u];
#pragma unroll
          for (int u = 0; u < 3; ++u) *reinterpret_cast<float4 *>(&pv[4 * u]) = p4[u];
#pragma unroll
          for (int cc = 0; cc < 9; ++cc) {
            a0 = __fmaf_rn(rv[cc], pv[cc], a0);
            a1 = __fmaf_rn(rv[9 + cc], pv[cc], a1);
            a2 = __fmaf_rn(rv[18 + cc], pv[cc], a2);
          }
        }
      } else {
        const int r0 = B.sblk_row[c], nb = B.sblk_row[c + 1] - r0;
        for (int v = lane; v <= nb; v += kClSub) {
          const float *row = (v < nb ? vals + 81 * (size_t)(r0 + v) : Sii + 81 * (size_t)c) + 9 * g;
          const float *pc = ph + 12 * ((v < nb ? B.sblk_col[r0 + v] : c) - c0);
#pragma unroll
          for (int cc = 0; cc < 9; ++cc) {
            const float pv = pc[cc];
            a0 = __fmaf_rn(row[cc], pv, a0);
            a1 = __fmaf_rn(row[27 + cc], pv, a1);
            a2 = __fmaf_rn(row[54 + cc], pv, a2);
          }
        }
      }
      // the sums of the three rows over the group's lanes, the xor tree 1, 2,
      // 4 of each row with its additions spread over the lanes: the first
      // level adds plain floats (an exact TwoSum), the later ones are done in
      // lanes 0, 1 and 2 (and their xor-4 twins) for rows g, g + 3 and g + 6
      // (lane 3 repeats lane 2's)
      const DF e0 = df_two_sum(a0, __shfl_xor_sync(gmask, a0, 1));
      const DF e1 = df_two_sum(a1, __shfl_xor_sync(gmask, a1, 1));
      const DF e2 = df_two_sum(a2, __shfl_xor_sync(gmask, a2, 1));
      const DF e01 = lane & 1 ? e1 : e0;
      DF d = lane & 2 ? e2 : e01;
      const DF give = lane & 2 ? e01 : e2;  // the row of the lane's xor-2 partner
      d = df_add(d, DF{__shfl_xor_sync(gmask, give.hi, 2), __shfl_xor_sync(gmask, give.lo, 2)});
      d = df_add(d, DF{__shfl_xor_sync(gmask, d.hi, 4), __shfl_xor_sync(gmask, d.lo, 4)});
      if (lane < 3) {
        const int i = 9 * lc + g + 3 * lane;
        qh[i] = d.hi, ql[i] = d.lo;
      }
    }
    __syncthreads();
    // each owned camera's p.q
    for (int cb = 0; cb + wc < own_n; cb += T / 16) {
      const int lc = cb + hc;
      DF d = df_zero();
      if (lc < own_n && hq < 9) {
        const int i = 9 * lc + hq;
        d = df_mul_f(DF{qh[i], ql[i]}, ph[12 * (own0 + lc) + hq]);
      }
      d = df_group16_sum(d, hmask);
      if (lc < own_n && hq == 0) cpq[own0 + lc] = make_float2(d.hi, d.lo);
    }
    if (cs > 1) {
      __syncwarp();
      cluster_arrive(), cluster_wait();
      // 2. p.q, alpha, the owned update
      // the other CTAs' cameras' values, read from their shared memory
      for (int c = t; c < n; c += T) {
        const int r = own_of[c];
        if (r != rank) cpq[c] = *peer(cpq + c, r);
      }
    }
    __syncthreads();
    if (t < 32) {
      const DF s = cam_total(cpq, 1, n);
      if (t == 0) scf[0] = s;
    }
    __syncthreads();
    const DF pq = scf[0];
    if (!(pq.hi > 0.f && isfinite(pq.hi))) {  // S not positive definite along p_k: the PCG ends with x_k
      if (k == 0) linear_ok = false;
      break;
    }
    const DF alpha = df_div(rz, pq);
    const DF nalpha = df_neg(alpha);
    auto step_x = [&](int i, int ip) {
      const DF x = df_add(DF{xh[i], xl[i]}, df_mul_f(alpha, ph[ip]));
      xh[i] = x.hi, xl[i] = x.lo;
      return x;
    };
    for (int cb = 0; cb + wc < own_n; cb += T / 16) {
      const int lc = cb + hc;
      const bool act = lc < own_n && hq < 9;
      const int i = 9 * lc + hq;
      DF r = df_zero();
      if (act) {
        r = df_add(DF{rh[i], rl[i]}, df_mul(nalpha, DF{qh[i], ql[i]}));
        rh[i] = r.hi, rl[i] = r.lo;
      }
      __syncwarp(hmask);  // the camera's r, for z = M r
      DF d0 = df_zero(), d1 = df_zero(), d2 = df_zero();
      if (act) {
        const float *m = Mo + 81 * lc + 9 * hq;
        const float *rr = rh + 9 * lc;
        float u = 0.f;
#pragma unroll
        for (int kk = 0; kk < 9; ++kk) u = __fmaf_rn(m[kk], rr[kk], u);
        zf[a9 + i] = u;
        d0 = df_mul_f(r, u);
        d1 = df_mul(r, r);
        if (QUAD) d2 = df_mul(step_x(i, 12 * (own0 + lc) + hq), df_add(DF{vh[i], vl[i]}, r));
      }
      // both sums in one tree: from the first level on the even lanes add up
      // r.z, the odd ones r.r
      const bool odd = (hq & 1) != 0;
      const DF give = odd ? d0 : d1;
      DF d = df_add(odd ? d1 : d0, DF{__shfl_xor_sync(hmask, give.hi, 1), __shfl_xor_sync(hmask, give.lo, 1)});
#pragma unroll
      for (int off = 2; off < 16; off <<= 1)
        d = df_add(d, DF{__shfl_xor_sync(hmask, d.hi, off), __shfl_xor_sync(hmask, d.lo, off)});
      if (lc < own_n && hq < 2) reinterpret_cast<float2 *>(crr)[2 * (own0 + lc) + hq] = make_float2(d.hi, d.lo);
      if (QUAD) {
        d2 = df_group16_sum(d2, hmask);
        if (lc < own_n && hq == 0) cxv[own0 + lc] = make_float2(d2.hi, d2.lo);
      }
    }
    __syncwarp();
    if (cs > 1) cluster_arrive();
    // x is nobody's input until the end (unless the stopping test takes it)
    if (!QUAD)
      for (int i = t; i < o9; i += T) step_x(i, 12 * own0 + i + 3 * (i / 9));
    __syncwarp();
    // 3. the stopping test on (x_{k+1}, r_{k+1}) and beta_{k+1}: the other
    // CTAs' cameras' values, then warps 0-2 sum them while the others read the
    // other CTAs' z (both from the owners' shared memory)
    if (cs > 1) {
      cluster_wait();
      for (int c = t; c < n; c += T) {
        const int r = own_of[c];
        if (r != rank) {
          crr[c] = *peer(crr + c, r);
          if (QUAD) cxv[c] = *peer(cxv + c, r);
        }
      }
    }
    __syncthreads();
    if (t < 96) {  // warps 0, 1, 2: r.z, r.r, x.(v + r)
      const int j = t >> 5;
      const float2 *v = reinterpret_cast<const float2 *>(crr);
      if (j < 2 || QUAD) {
        const DF sj = cam_total(j < 2 ? v + j : cxv, j < 2 ? 2 : 1, n);
        if ((t & 31) == 0) scf[1 + j] = sj;
      }
    } else if (cs > 1) {
      for (int i = i_lo + t - 96; i < i_hi; i += T - 96) {
        const int r = own_of[i / 9];
        if (r != rank) zf[i] = *peer(zf + i, r);
      }
    }
    __syncthreads();
    // every thread takes the same decision from the same values
    const DF rz1 = scf[1], rr1 = scf[2];
    const int k1 = k + 1;
    bool stop = false;
    if (QUAD) {
      const double qk = -df_value(scf[3]);  // Q(x) = x'Sx - 2 v'x = -x.(v + r)
      const double lhs = k1 * (qk - q0), rhs = o.eta * qk;
      const bool below = qk > 0.0 ? lhs < rhs : (qk < 0.0 ? lhs > rhs : q0 > 0.0);
      if (below && k1 >= o.min_pcg_iterations) stop = true;
      q0 = qk;
    } else if (df_le(rr1, lim2) && k1 >= o.min_pcg_iterations) {
      stop = true;
    }
    if (k1 >= o.max_pcg_iterations) stop = true;
    if (!(rz1.hi != 0.f && isfinite(rz1.hi))) stop = true;
    const DF beta = df_div(rz1, rz);
    last_beta = beta;
    last_rr = rr1;
    rz = rz1;
    last_pq = pq;
    ++k;
    if (stop) break;
    // p_{k+1} = z_{k+1} + beta p_k, rounded once to FP32
    for (int i = i_lo + t; i < i_hi; i += T) {
      const int ip = i + 3 * (i / 9);
      ph[ip] = df_add(DF{zf[i], 0.f}, df_mul_f(beta, ph[ip])).hi;
    }
    __syncthreads();
  }
  __syncthreads();  // x of every thread
  // results: the owned x (the camera step) and the PCG vectors; the state
  for (int i = t; i < o9; i += T) {
    const size_t gi = g0 + a9 + i;
    B.pcg_x[gi] = df_value(DF{xh[i], xl[i]});
    B.pcg_r[gi] = df_value(DF{rh[i], rl[i]});
    B.pcg_z[gi] = (double)zf[a9 + i];
    B.pcg_p[gi] = (double)ph[12 * own0 + i + 3 * (i / 9)];
  }
  if (rank == 0 && t == 0) {
    L->pcg_iterations = k;
    if (!linear_ok) L->linear_ok = 0;
    if (k > 0) {
      L->beta = df_value(last_beta);
      L->rz = df_value(rz);
      L->rr = df_value(last_rr);
      L->q0 = q0;
      L->pq = df_value(last_pq);
    }
    L->pcg_active = 0;
  }
  // no CTA leaves before the others have read what it stored for them
  __syncwarp();
  if (cs > 1) cluster_arrive(), cluster_wait();
}

static const void *cluster_kernel(bool quad) {
  return quad ? (const void *)k_pcg_cluster<true> : (const void *)k_pcg_cluster<false>;
}

bool pcg_cluster_plan(const ProblemInfo *prob, int num_problems, const int32_t *sblk_row, int cams_per_cta, bool quad,
                      int running, ClusterPlan *plan) {
  *plan = ClusterPlan();
  const void *kernel = cluster_kernel(quad);
  int n_max = 0;
  for (int p = 0; p < num_problems; ++p) n_max = std::max(n_max, (int)prob[p].cam_count);
  if (n_max <= 0 || n_max > kClMaxCams) return false;
  int dev = 0, sms = 0, optin = 0, per_sm_bytes = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&per_sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (sms <= 0) return false;
  int cs_only = 0;  // the tuned split: the smallest cluster of at most cams_per_cta cameras a CTA
  if (cams_per_cta > 0)
    for (cs_only = 1; cs_only < kClMaxCS && (n_max + cs_only - 1) / cs_only > cams_per_cta;) cs_only *= 2;
  // The cluster size and the CTA's threads with the shortest estimated PCG
  // iteration of the largest problem, in clocks, times the CTAs that an SM
  // runs one after the other: the product, bound by the shared-memory reads
  // of S (7.5 clocks per block; from L2 when the rows do not fit), its rounds
  // and the update's over the CTA's threads, and the rest of the chain (two
  // cluster barriers and their read-backs, about 2,200 clocks, when cs > 1).
  // Measured, the PCG of an LM iteration (100 iterations), cs / threads: one
  // window of 23 cameras 1/512 375 us, 2/256 424, 4/256 365, 8/256 354; 48
  // windows of 5-40 cameras 1/512 605, 2/512 479, 4/256 485, 8/256 742; 192
  // windows 1/512 934, 2/256 994, 4/256 1,284; 256 windows of 7 cameras 1/256
  // 114, 1/512 206; 250 cameras 16/256 696, 16/512 606.
  double best = 1e300;
  ClLayout l{};
  int cs = 0, own = 0, cache = 0, threads = 0;
  for (int c2 = 1; c2 <= kClMaxCS; c2 *= 2) {
    if (cs_only > 0 && c2 != cs_only) continue;
    // the kernel's split of each problem's cameras (runs of about equal
    // blocks): the largest run and its blocks
    int o2 = 0, mb = 0;
    for (int p = 0; p < num_problems; ++p) {
      const int n = prob[p].cam_count, c0 = prob[p].cam_begin, r0 = sblk_row[c0];
      const long long wtot = (long long)(sblk_row[c0 + n] - r0) + n;
      int a = 0;
      for (int r = 0; r < c2; ++r) {
        const long long tb = ((long long)(r + 1) * wtot + c2 - 1) / c2;
        int b = a;
        while (b < n && (long long)(sblk_row[c0 + b] - r0) + b < tb) ++b;
        o2 = std::max(o2, b - a);
        mb = std::max(mb, (int)(sblk_row[c0 + b] - sblk_row[c0 + a]) + (b - a));
        a = b;
      }
    }
    if (o2 > kClMaxOwn) continue;
    for (int ca = 1; ca >= 0; --ca) {
      const ClLayout l2 = cl_layout(n_max, o2, ca ? mb : 0);
      if (l2.total > (size_t)optin) continue;
      for (int th : {256, 512}) {
        const int occ = std::max(1, std::min(512 / th, (int)((size_t)per_sm_bytes / (l2.total + 1024))));  // (128 registers a thread)
        const double load = (double)running * c2 / sms;
        const double waves = load <= occ ? 1.0 : load / occ + 0.25, share = load > 1.0 && occ > 1 ? 1.15 : 1.0;
        const double rounds = std::ceil(3.0 * o2 / (th / 8)), upd = std::ceil((double)o2 / (th / 16));
        const double est = waves * share * ((ca ? 7.5 : 32.0) * mb + 500.0 * rounds + (th == 256 ? 1100.0 : 1500.0) * upd +
                                            400.0 * (th / 256) + (c2 > 1 ? 5200.0 : 3000.0));
        if (est < best) best = est, cs = c2, own = o2, cache = ca ? mb : 0, threads = th, l = l2;
      }
    }
  }
  if (cs == 0) return false;
  if (raise_smem_limit(kernel, l.total) != cudaSuccess ||
      (cs > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = l.total;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return false;
  }
  plan->cs = cs;
  plan->n_max = n_max;
  plan->own_max = own;
  plan->threads = threads;
  plan->quad = quad;
  plan->cache_blocks = cache;
  plan->smem = l.total;
  return true;
}

cudaError_t launch_pcg_cluster(const DeviceBatch &b, const ClusterPlan &plan, cudaStream_t s) {
  if (b.num_problems == 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(b.num_problems * plan.cs));
  cfg.blockDim = dim3((unsigned)plan.threads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)plan.cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, plan.quad ? k_pcg_cluster<true> : k_pcg_cluster<false>, b, plan.cs, plan.n_max,
                            plan.own_max, plan.cache_blocks, plan.above, plan.upto);
}

}  // namespace gba
