// FP64 vector kernels for the PCG recurrence (saige-linalg/src/
// decomposition.rs:212-298), the fit-null operator and Jacobi preconditioner
// (saige-core/src/glmm/ai_reml.rs:142-164) and the AI-REML elementwise work
// (family.rs, link.rs).  Reductions are two-stage with a partition fixed by n,
// so every result is deterministic from run to run.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "kernels_vec.cuh"
#include "rng.hpp"

namespace saige {

namespace {

namespace cg = cooperative_groups;

constexpr int kT = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) {
    for (int k = 0; k < kT / 32; ++k) s += sh[k];
  }
  __syncthreads();
  return s;  // valid in thread 0
}

__device__ __forceinline__ int64_t part_chunk(int64_t n) {
  return (n + gridDim.x - 1) / gridDim.x;
}

// Sum nb partials of k quantities per column in a fixed order; one warp per
// (column, quantity).
__global__ void reduce_partials(const double* __restrict__ partial, int nb, int nq,
                                double* __restrict__ out) {
  const int idx = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (idx >= nq) return;
  const int l = threadIdx.x & 31;
  double s = 0.0;
  for (int b = l; b < nb; b += 32) s += partial[(int64_t)idx * nb + b];
  s = warp_sum(s);
  if (l == 0) out[idx] = s;
}

__global__ void col_dots_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                int64_t n, int64_t ld, double* __restrict__ partial) {
  __shared__ double sh[kT / 32];
  const int c = blockIdx.y;
  const int64_t ch = part_chunk(n), lo = (int64_t)blockIdx.x * ch;
  int64_t hi = lo + ch;
  if (hi > n) hi = n;
  const double* ac = a + (int64_t)c * ld;
  const double* bc = b + (int64_t)c * ld;
  double s = 0.0;
  for (int64_t i = lo + threadIdx.x; i < hi; i += kT) s += ac[i] * bc[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partial[(int64_t)c * gridDim.x + blockIdx.x] = s;
}

__global__ void cross_dots_kernel(const double* __restrict__ a, const double* __restrict__ b,
                                  int q, const double* __restrict__ w, int64_t n, int64_t ld,
                                  double* __restrict__ partial) {
  __shared__ double sh[kT / 32];
  const int pair = blockIdx.y;
  const int j = pair / q, k = pair % q;
  const int64_t ch = part_chunk(n), lo = (int64_t)blockIdx.x * ch;
  int64_t hi = lo + ch;
  if (hi > n) hi = n;
  const double* aj = a + (int64_t)j * ld;
  const double* bk = b + (int64_t)k * ld;
  double s = 0.0;
  if (w) {
    for (int64_t i = lo + threadIdx.x; i < hi; i += kT) s += aj[i] * w[i] * bk[i];
  } else {
    for (int64_t i = lo + threadIdx.x; i < hi; i += kT) s += aj[i] * bk[i];
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partial[(int64_t)pair * gridDim.x + blockIdx.x] = s;
}

// The PCG kernels' elementwise loops are bound by the latency of their loads: at n = 9,001 a
// column has three blocks (the partition fixes the order of its sums), and a thread eleven
// rows.  It takes kPcgBatch rows at a time, all loads before the first use, and adds to its
// sums in row order as before (31 columns of 9,001: pcg_update 23.8 -> 8.2 us,
// pcg_apply 11.7 -> 4.9, pcg_start 8.4 -> 5.5).  The sums over the blocks are formed by the
// kernel that needs them, in every block alike, instead of a launch each (2.4 and 1.8 us, and
// their gaps; pcg_p 2.3 -> 4.6).
constexpr int kPcgBatch = 4;

// Into sh, for every thread of the block: the sums of nb partials of up to three quantities
// (NULL: none), a warp each, in the order of reduce_partials.
__device__ __forceinline__ void block_partials(const double* a, const double* b, const double* c,
                                               int nb, double* sh) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const double* from = w == 0 ? a : (w == 1 ? b : (w == 2 ? c : nullptr));
  if (from) {
    double s = 0.0;
    for (int k = l; k < nb; k += 32) s += from[k];
    s = warp_sum(s);
    if (l == 0) sh[w] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kT)
    pcg_start_kernel(const double* __restrict__ b, const double* __restrict__ x0,
                     const double* __restrict__ ax0, const double* __restrict__ d,
                     double* __restrict__ x, double* __restrict__ r, double* __restrict__ z,
                     double* __restrict__ p, int64_t n, int64_t ld,
                     double* __restrict__ partial) {
  __shared__ double sh[kT / 32];
  const int c = blockIdx.y;
  const int64_t off = (int64_t)c * ld;
  const int64_t ch = part_chunk(n), lo = (int64_t)blockIdx.x * ch;
  int64_t hi = lo + ch;
  if (hi > n) hi = n;
  double s_rz = 0.0, s_rr = 0.0, s_bb = 0.0;
  for (int64_t i0 = lo + threadIdx.x; i0 < hi; i0 += kPcgBatch * kT) {
    double bi[kPcgBatch], xi[kPcgBatch], ai[kPcgBatch], di[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      bi[k] = in ? b[off + i] : 0.0;
      xi[k] = in && x0 ? x0[off + i] : 0.0;
      ai[k] = in && ax0 ? ax0[off + i] : 0.0;
      di[k] = in ? d[i] : 1.0;
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      if (i >= hi) break;
      const double ri = bi[k] - ai[k];
      const double zi = ri / di[k];
      x[off + i] = xi[k];
      r[off + i] = ri;
      z[off + i] = zi;
      p[off + i] = zi;
      s_rz += ri * zi;
      s_rr += ri * ri;
      s_bb += bi[k] * bi[k];
    }
  }
  const int nb = gridDim.x, q = gridDim.y;
  s_rz = block_sum(s_rz, sh);
  s_rr = block_sum(s_rr, sh);
  s_bb = block_sum(s_bb, sh);
  if (threadIdx.x == 0) {
    partial[((int64_t)0 * q + c) * nb + blockIdx.x] = s_rz;
    partial[((int64_t)1 * q + c) * nb + blockIdx.x] = s_rr;
    partial[((int64_t)2 * q + c) * nb + blockIdx.x] = s_bb;
  }
}

__device__ __forceinline__ void pcg_first_state(int c, double rz, double rr, double bb, double tol,
                                                int force_step, const PcgCols& cols) {
  const double bn = sqrt(bb);
  const double tol_abs = tol * (bn > 1.0 ? bn : 1.0);
  cols.rz[c] = rz;
  cols.rr[c] = rr;
  cols.tol_abs[c] = tol_abs;
  cols.iters[c] = 0;
  // a warm-started column takes at least one CG step (force_step), so a start
  // that already meets the tolerance is still refined against the current operator
  cols.state[c] = (!force_step && sqrt(rr) < tol_abs) ? kColConverged : kColActive;
}

__global__ void pcg_start_finish(const double* __restrict__ sums, int q, double tol, int force_step,
                                 PcgCols cols, unsigned int* __restrict__ tickets) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= q) return;
  tickets[c] = 0u;
  pcg_first_state(c, sums[c], sums[q + c], sums[2 * q + c], tol, force_step, cols);
}

template <bool kWInverse>
__global__ void __launch_bounds__(kT)
    pcg_apply_kernel(const double* __restrict__ p, const double* __restrict__ kp,
                     const double* __restrict__ wv, double tau0, double tau1,
                     double* __restrict__ ap, int64_t n, int64_t ld,
                     const int32_t* __restrict__ state, double* __restrict__ partial) {
  __shared__ double sh[kT / 32];
  const int c = blockIdx.y;
  if (state[c] != kColActive) return;
  const int64_t off = (int64_t)c * ld;
  const int64_t ch = part_chunk(n), lo = (int64_t)blockIdx.x * ch;
  int64_t hi = lo + ch;
  if (hi > n) hi = n;
  double s = 0.0;
  for (int64_t i0 = lo + threadIdx.x; i0 < hi; i0 += kPcgBatch * kT) {
    double pk[kPcgBatch], kk[kPcgBatch], wk[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      pk[k] = in ? p[off + i] : 0.0;
      kk[k] = in ? kp[off + i] : 0.0;
      wk[k] = in ? wv[i] : 1.0;
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      if (i >= hi) break;
      const double pi = pk[k];
      // ai_reml.rs:147 (tau0 v / max(w,1e-30) + tau1 Kv) or pcg.rs:56 (tau0 w v + tau1 Kv)
      const double a = kWInverse ? tau0 * pi / wk[k] + tau1 * kk[k]
                                 : tau0 * wk[k] * pi + tau1 * kk[k];
      ap[off + i] = a;
      s += pi * a;
    }
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partial[(int64_t)c * gridDim.x + blockIdx.x] = s;
}

// pap: pcg_apply's partials, whose sums every block forms for itself.  A column with |pap| <
// 1e-30 stops (decomposition.rs:257-264): pcg_p_kernel says so.
__global__ void __launch_bounds__(kT)
    pcg_update_kernel(double* __restrict__ x, double* __restrict__ r, double* __restrict__ z,
                      const double* __restrict__ p, const double* __restrict__ ap,
                      const double* __restrict__ d, int64_t n, int64_t ld, PcgCols cols,
                      const double* __restrict__ pap_partial, double* __restrict__ partial,
                      double* __restrict__ kx, const double* __restrict__ kp) {
  __shared__ double sh[kT / 32];
  const int c = blockIdx.y;
  const int nb = gridDim.x, q = gridDim.y;
  if (cols.state[c] != kColActive) return;
  block_partials(pap_partial + (int64_t)c * nb, nullptr, nullptr, nb, sh);
  const double pap = sh[0];
  if (fabs(pap) < 1e-30) return;
  __syncthreads();  // sh is free again
  const double alpha = cols.rz[c] / pap;
  const int64_t off = (int64_t)c * ld;
  const int64_t ch = part_chunk(n), lo = (int64_t)blockIdx.x * ch;
  int64_t hi = lo + ch;
  if (hi > n) hi = n;
  double s_rz = 0.0, s_rr = 0.0;
  for (int64_t i0 = lo + threadIdx.x; i0 < hi; i0 += kPcgBatch * kT) {
    double pk[kPcgBatch], xk[kPcgBatch], rk[kPcgBatch], ak[kPcgBatch], dk[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      pk[k] = in ? p[off + i] : 0.0;
      xk[k] = in ? x[off + i] : 0.0;
      rk[k] = in ? r[off + i] : 0.0;
      ak[k] = in ? ap[off + i] : 0.0;
      dk[k] = in ? d[i] : 1.0;
    }
    if (kx) {  // K x follows x: K x += alpha K p
      double kxk[kPcgBatch], kpk[kPcgBatch];
#pragma unroll
      for (int k = 0; k < kPcgBatch; ++k) {
        const int64_t i = i0 + k * kT;
        kxk[k] = i < hi ? kx[off + i] : 0.0;
        kpk[k] = i < hi ? kp[off + i] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < kPcgBatch; ++k) {
        const int64_t i = i0 + k * kT;
        if (i < hi) kx[off + i] = kxk[k] + alpha * kpk[k];
      }
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      if (i >= hi) break;
      x[off + i] = xk[k] + alpha * pk[k];
      const double ri = rk[k] - alpha * ak[k];
      r[off + i] = ri;
      const double zi = ri / dk[k];
      z[off + i] = zi;
      s_rz += ri * zi;
      s_rr += ri * ri;
    }
  }
  s_rz = block_sum(s_rz, sh);
  s_rr = block_sum(s_rr, sh);
  if (threadIdx.x == 0) {
    partial[((int64_t)0 * q + c) * nb + blockIdx.x] = s_rz;
    partial[((int64_t)1 * q + c) * nb + blockIdx.x] = s_rr;
  }
}

// p = z + beta p of the columns that go on.  Every block forms beta and the next state from
// the nb partials of pcg_apply and pcg_update; the one that takes the column's last ticket,
// when no block reads the old ones any more, writes them.
__global__ void __launch_bounds__(kT)
    pcg_p_kernel(double* __restrict__ p, const double* __restrict__ z, int64_t n, int64_t ld,
                 const double* __restrict__ pap_partial, const double* __restrict__ partial,
                 int nb, int max_iter, PcgCols cols, unsigned int* __restrict__ tickets) {
  __shared__ double sh[3];
  const int c = blockIdx.y, q = gridDim.y;
  if (cols.state[c] != kColActive) return;
  block_partials(partial + ((int64_t)0 * q + c) * nb, partial + ((int64_t)1 * q + c) * nb,
                 pap_partial + (int64_t)c * nb, nb, sh);
  const double s_rz = sh[0], s_rr = sh[1];
  const bool stop = fabs(sh[2]) < 1e-30;  // (pcg_update left no sums of such a column)
  const double beta = s_rz / cols.rz[c];
  const int it = cols.iters[c] + 1;
  const int next = stop                            ? kColStopped
                   : sqrt(s_rr) < cols.tol_abs[c] ? kColConverged
                   : it >= max_iter               ? kColMaxIter
                                                  : kColActive;
  if (next == kColActive) {
    const int64_t off = (int64_t)c * ld;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
      p[off + i] = z[off + i] + beta * p[off + i];
  }
  __syncthreads();  // the block has read the column's scalars
  if (threadIdx.x != 0) return;
  if (atomicAdd(&tickets[c], 1u) != gridDim.x - 1) return;
  tickets[c] = 0u;
  cols.state[c] = next;
  if (stop) return;
  cols.rz[c] = s_rz;
  cols.rr[c] = s_rr;
  cols.iters[c] = it;
}

// Columns of up to kClusterRows row blocks: a cluster per column, a thread block per row block,
// whose sums are those of the kernels above in the same order: each block's partial sum, then
// a warp over the blocks' (read through distributed shared memory) as in reduce_partials.  A
// whole PCG iteration is then one launch, a, then z, kept in shared memory: 31 columns of 9,001
// in 14.0 us against 17.7 in three launches (17.1 with one thread block of 768 threads per
// column: one SM's bandwidth); dot products and their sum 4.3 us against 3.6 + 1.7.
constexpr int kClusterRows = 8;  // the portable cluster size

// The barrier of a column's blocks (a column of one row block is launched without a cluster).
__device__ __forceinline__ void column_barrier() {
  if (gridDim.x > 1)
    cg::this_cluster().sync();
  else
    __syncthreads();
}

// The sums of up to kQ quantities over the cluster, in every thread.  part must not be written
// again before a later cluster barrier.  sh: kQ x 9 doubles.
template <int kQ>
__device__ __forceinline__ void column_sums(double (&v)[kQ], double* sh, double* part) {
  const cg::cluster_group cl = cg::this_cluster();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kQ; ++k) {
    v[k] = warp_sum(v[k]);
    if (l == 0) sh[k * 9 + w] = v[k];
  }
  __syncthreads();
  if (w < kQ && l == 0) {
    double s = 0.0;
    for (int k = 0; k < kT / 32; ++k) s += sh[w * 9 + k];
    part[w] = s;
  }
  column_barrier();
  if (w < kQ) {
    double s = 0.0;
    if (l < (int)gridDim.x) s += gridDim.x > 1 ? *cl.map_shared_rank(part + w, l) : part[w];
    s = warp_sum(s);
    if (l == 0) sh[w * 9 + 8] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kQ; ++k) v[k] = sh[k * 9 + 8];
}

// This thread's rows [lo, hi), every kT-th, of the block's row block.
__device__ __forceinline__ void column_rows(int64_t n, int64_t& lo, int64_t& hi) {
  const int64_t ch = part_chunk(n), from = (int64_t)blockIdx.x * ch;
  hi = from + ch < n ? from + ch : n;
  lo = from + threadIdx.x;
}

template <bool kWInverse>
__global__ void __launch_bounds__(kT)
    pcg_iteration_kernel(double* __restrict__ x, double* __restrict__ r, double* __restrict__ p,
                         const double* __restrict__ kp, const double* __restrict__ wv,
                         double tau0, double tau1, const double* __restrict__ d, int64_t n,
                         int64_t ld, int max_iter, PcgCols cols, double* __restrict__ kx,
                         const PcgSeen seen) {
  extern __shared__ double az[];  // the row block's a = (Sigma p), then z
  __shared__ double sh[2 * 9], part[3];
  const int c = blockIdx.y;
  const int64_t first = (int64_t)blockIdx.x * part_chunk(n);
  if (cols.state[c] != kColActive) return;
  const int64_t off = (int64_t)c * ld;
  int64_t lo, hi;
  column_rows(n, lo, hi);
  double pap[1] = {0.0};
  for (int64_t i0 = lo; i0 < hi; i0 += kPcgBatch * kT) {
    double pk[kPcgBatch], kk[kPcgBatch], wk[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      pk[k] = in ? p[off + i] : 0.0;
      kk[k] = in ? kp[off + i] : 0.0;
      wk[k] = in ? wv[i] : 1.0;
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      if (i >= hi) break;
      const double pi = pk[k];
      const double a = kWInverse ? tau0 * pi / wk[k] + tau1 * kk[k]
                                 : tau0 * wk[k] * pi + tau1 * kk[k];
      az[i - first] = a;
      pap[0] += pi * a;
    }
  }
  column_sums(pap, sh, part);
  if (fabs(pap[0]) < 1e-30) {  // decomposition.rs:257-264
    column_barrier();  // every block has read the partial sums and the column's state
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      cols.state[c] = kColStopped;
      if (seen.state) seen.state[c] = kColStopped;
    }
    return;
  }
  const double rz = cols.rz[c], alpha = rz / pap[0];
  double sums[2] = {0.0, 0.0};
  for (int64_t i0 = lo; i0 < hi; i0 += kPcgBatch * kT) {
    double pk[kPcgBatch], xk[kPcgBatch], rk[kPcgBatch], dk[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      pk[k] = in ? p[off + i] : 0.0;
      xk[k] = in ? x[off + i] : 0.0;
      rk[k] = in ? r[off + i] : 0.0;
      dk[k] = in ? d[i] : 1.0;
    }
    if (kx) {  // K x follows x: K x += alpha K p
      double kxk[kPcgBatch], kpk[kPcgBatch];
#pragma unroll
      for (int k = 0; k < kPcgBatch; ++k) {
        const int64_t i = i0 + k * kT;
        kxk[k] = i < hi ? kx[off + i] : 0.0;
        kpk[k] = i < hi ? kp[off + i] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < kPcgBatch; ++k) {
        const int64_t i = i0 + k * kT;
        if (i < hi) kx[off + i] = kxk[k] + alpha * kpk[k];
      }
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      if (i >= hi) break;
      x[off + i] = xk[k] + alpha * pk[k];
      const double ri = rk[k] - alpha * az[i - first];
      r[off + i] = ri;
      const double zi = ri / dk[k];
      az[i - first] = zi;
      sums[0] += ri * zi;
      sums[1] += ri * ri;
    }
  }
  __syncthreads();  // sh is free again
  column_sums(sums, sh, part + 1);
  const int it = cols.iters[c] + 1;
  const int next = sqrt(sums[1]) < cols.tol_abs[c] ? kColConverged
                   : it >= max_iter               ? kColMaxIter
                                                  : kColActive;
  const double beta = sums[0] / rz;
  if (next == kColActive) {
    for (int64_t i0 = lo; i0 < hi; i0 += kPcgBatch * kT) {
      double pk[kPcgBatch];
#pragma unroll
      for (int k = 0; k < kPcgBatch; ++k) pk[k] = i0 + k * kT < hi ? p[off + i0 + k * kT] : 0.0;
#pragma unroll
      for (int k = 0; k < kPcgBatch; ++k) {
        const int64_t i = i0 + k * kT;
        if (i < hi) p[off + i] = az[i - first] + beta * pk[k];
      }
    }
  }
  column_barrier();  // every block has read the partial sums and the column's scalars
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cols.rz[c] = sums[0];
    cols.rr[c] = sums[1];
    cols.iters[c] = it;
    cols.state[c] = next;
    if (seen.state) {
      seen.rr[c] = sums[1];
      seen.iters[c] = it;
      seen.state[c] = next;
    }
  }
}

// pcg_start_kernel, the sums and pcg_start_finish in one.
__global__ void __launch_bounds__(kT)
    pcg_start_column_kernel(const double* __restrict__ b, const double* __restrict__ x0,
                            const double* __restrict__ ax0, const double* __restrict__ d,
                            double* __restrict__ x, double* __restrict__ r,
                            double* __restrict__ p, int64_t n, int64_t ld, double tol,
                            int force_step, PcgCols cols, const PcgSeen seen) {
  __shared__ double sh[3 * 9], part[3];
  const int c = blockIdx.y;
  const int64_t off = (int64_t)c * ld;
  int64_t lo, hi;
  column_rows(n, lo, hi);
  double sums[3] = {0.0, 0.0, 0.0};
  for (int64_t i0 = lo; i0 < hi; i0 += kPcgBatch * kT) {
    double bi[kPcgBatch], xi[kPcgBatch], ai[kPcgBatch], di[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      bi[k] = in ? b[off + i] : 0.0;
      xi[k] = in && x0 ? x0[off + i] : 0.0;
      ai[k] = in && ax0 ? ax0[off + i] : 0.0;
      di[k] = in ? d[i] : 1.0;
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      if (i >= hi) break;
      const double ri = bi[k] - ai[k];
      const double zi = ri / di[k];
      x[off + i] = xi[k];
      r[off + i] = ri;
      p[off + i] = zi;
      sums[0] += ri * zi;
      sums[1] += ri * ri;
      sums[2] += bi[k] * bi[k];
    }
  }
  column_sums(sums, sh, part);
  column_barrier();  // the partial sums are read
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    pcg_first_state(c, sums[0], sums[1], sums[2], tol, force_step, cols);
    if (seen.state) {
      seen.rr[c] = sums[1];
      seen.iters[c] = 0;
      seen.state[c] = cols.state[c];
    }
  }
}

// out[column or pair] in one launch: col_dots_kernel or cross_dots_kernel and reduce_partials.
__global__ void __launch_bounds__(kT)
    dots_column_kernel(const double* __restrict__ a, const double* __restrict__ b, int q,
                       bool cross, const double* __restrict__ w, int64_t n, int64_t ld,
                       double* __restrict__ out) {
  __shared__ double sh[9], part[1];
  const int pair = blockIdx.y, ja = cross ? pair / q : pair, jb = cross ? pair % q : pair;
  const double* aj = a + (int64_t)ja * ld;
  const double* bk = b + (int64_t)jb * ld;
  int64_t lo, hi;
  column_rows(n, lo, hi);
  double s[1] = {0.0};
  for (int64_t i0 = lo; i0 < hi; i0 += kPcgBatch * kT) {
    double x[kPcgBatch], y[kPcgBatch], v[kPcgBatch];
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      const int64_t i = i0 + k * kT;
      const bool in = i < hi;
      x[k] = in ? aj[i] : 0.0;
      y[k] = in ? bk[i] : 0.0;
      v[k] = in && w ? w[i] : 1.0;
    }
#pragma unroll
    for (int k = 0; k < kPcgBatch; ++k) {
      if (i0 + k * kT >= hi) break;
      if (w)
        s[0] += x[k] * v[k] * y[k];
      else
        s[0] += x[k] * y[k];
    }
  }
  column_sums(s, sh, part);
  column_barrier();  // the partial sums are read
  if (blockIdx.x == 0 && threadIdx.x == 0) out[pair] = s[0];
}

__global__ void sigma_diag_kernel(const double* __restrict__ w, double tau0, double tau1,
                                  const double* __restrict__ diagk, double* __restrict__ wmax,
                                  double* __restrict__ d, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double wm = w[i] > 1e-30 ? w[i] : 1e-30;
  const double dg = diagk ? tau0 / wm + tau1 * diagk[i] : tau0 / wm + tau1;
  wmax[i] = wm;
  d[i] = fabs(dg) > 1e-30 ? dg : 1.0;
}

__global__ void sigma_diag_w_kernel(const double* __restrict__ w, double tau0, double tau1,
                                    double* __restrict__ d, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double dg = tau0 * w[i] + tau1;
  d[i] = fabs(dg) > 1e-30 ? dg : 1.0;
}

__device__ __forceinline__ double inv_link(int t, double eta) {
  if (t == SAIGE_TRAIT_BINARY) return 1.0 / (1.0 + exp(-eta));
  if (t == SAIGE_TRAIT_QUANTITATIVE) return eta;
  return 1.0 - exp(-exp(eta));
}

__global__ void eta_mu_kernel(const double* __restrict__ x, int p, const double* __restrict__ alpha,
                              int t, double* __restrict__ eta, double* __restrict__ mu, int64_t n,
                              int64_t ld) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // DenseMatrix::mat_vec column sweep order (dense.rs:102-113)
  double e = 0.0;
  for (int j = 0; j < p; ++j) e += x[(int64_t)j * ld + i] * alpha[j];
  eta[i] = e;
  double m = inv_link(t, e);
  if (t != SAIGE_TRAIT_QUANTITATIVE) {
    if (m < 1e-10) m = 1e-10;
    if (m > 1.0 - 1e-10) m = 1.0 - 1e-10;
  }
  mu[i] = m;
}

__global__ void work_vectors_kernel(const double* __restrict__ y, const double* __restrict__ eta,
                                    const double* __restrict__ mu, int t, double* __restrict__ w,
                                    double* __restrict__ ytil, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double m = mu[i];
  double v = t == SAIGE_TRAIT_QUANTITATIVE ? 1.0 : m * (1.0 - m);
  v = v > 1e-30 ? v : 1e-30;
  w[i] = v;
  if (ytil) {
    const double wm = v > 1e-30 ? v : 1e-30;
    ytil[i] = eta[i] + (y[i] - m) / wm;
  }
}

__global__ void init_mu_kernel(const double* __restrict__ y, int t, double* __restrict__ mu,
                               double* __restrict__ eta, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double yi = y[i];
  double m, e;
  if (t == SAIGE_TRAIT_BINARY) {
    m = (yi + 0.5) / 2.0;
    e = log(m / (1.0 - m));
  } else if (t == SAIGE_TRAIT_QUANTITATIVE) {
    m = yi;
    e = m;
  } else {
    m = (yi + 0.5) / 2.0;
    m = m < 0.01 ? 0.01 : (m > 0.99 ? 0.99 : m);
    e = log(-log(1.0 - m));
  }
  mu[i] = m;
  eta[i] = e;
}

// y = from - A coef (from may be y); rows n .. ld - 1 become from's.
__global__ void sub_combo_kernel(const double* from, double* y, int q,
                                 const double* __restrict__ a, int p,
                                 const double* __restrict__ coef, int64_t n, int64_t ld) {
  const int c = blockIdx.y;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ld) return;
  double v = from[(int64_t)c * ld + i];
  // ai_reml.rs:247-251: one subtraction per covariate column, in order
  if (i < n)
    for (int j = 0; j < p; ++j) v -= a[(int64_t)j * ld + i] * coef[j * q + c];
  y[(int64_t)c * ld + i] = v;
}

// t (p x q, row-major): each column's solve with the Cholesky factor l, with the host's
// operations in the host's order (decomposition.rs:64-89).  One chain of FP64 operations per
// column: 3.4 us for 3 covariates, 4.9 for 5, 11.8 for 11, in place of a read, a wait and a copy
// back.
__global__ void __launch_bounds__(64)
    chol_cols_kernel(const CholFactor l, int p, double* __restrict__ t, int q) {
  const int c = blockIdx.x * 64 + threadIdx.x;
  if (c >= q) return;
  double y[kCholMax];
  for (int i = 0; i < p; ++i) {
    double s = 0.0;
    for (int j = 0; j < i; ++j) s = __dadd_rn(s, __dmul_rn(l.v[i * p + j], y[j]));
    y[i] = __ddiv_rn(__dsub_rn(t[i * q + c], s), l.v[i * p + i]);
  }
  for (int i = p - 1; i >= 0; --i) {
    double s = 0.0;
    for (int j = i + 1; j < p; ++j) s = __dadd_rn(s, __dmul_rn(l.v[j * p + i], t[j * q + c]));
    t[i * q + c] = __ddiv_rn(__dsub_rn(y[i], s), l.v[i * p + i]);
  }
}

__global__ void div_w_kernel(const double* __restrict__ v, const double* __restrict__ w,
                             double* __restrict__ out, int64_t n, int64_t ld) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t off = (int64_t)blockIdx.y * ld;
  const double wm = w[i] > 1e-30 ? w[i] : 1e-30;
  out[off + i] = v[off + i] / wm;
}

// Column blockIdx.y of the list from two blocks of vectors to the slots from `slot` on.  One
// launch in place of two copies per column: the copies of five columns of 9,001 doubles took
// 1.9 us each on the device and longer to issue.
__global__ void __launch_bounds__(kT)
    keep_cols_kernel(const double* __restrict__ a, const double* __restrict__ b, KeepCols cols,
                     double* __restrict__ a_out, double* __restrict__ b_out, int slot,
                     int64_t ld) {
  const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;  // pairs of doubles (ld is even)
  if (2 * i >= ld) return;
  const int64_t from = (int64_t)cols.c[blockIdx.y] * ld + 2 * i;
  const int64_t to = (int64_t)(slot + blockIdx.y) * ld + 2 * i;
  const double2 x = *reinterpret_cast<const double2*>(a + from);
  const double2 y = *reinterpret_cast<const double2*>(b + from);
  *reinterpret_cast<double2*>(a_out + to) = x;
  *reinterpret_cast<double2*>(b_out + to) = y;
}

struct Key8 {
  uint32_t w[8];
};

// Rademacher probes from the ChaCha8 stream: word k = r * n + i (one block of 16
// words per thread) gives column r, sample i the value +1 when its sign bit is set
// (rand's gen::<bool>), else -1; rows n .. ld-1 of every column are zeroed.
__global__ void rademacher_kernel(Key8 key, int64_t n, int64_t ld, int nrv, double* __restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t words = (int64_t)nrv * n;
  if (c * 16 < words) {
    uint32_t w[16];
    chacha8_block(key.w, (uint64_t)c, w);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t k = c * 16 + j;
      if (k < words) {
        const int64_t r = k / n, i = k - r * n;
        out[r * ld + i] = static_cast<int32_t>(w[j]) < 0 ? 1.0 : -1.0;
      }
    }
  }
  // padding rows (ld - n per column)
  const int64_t pad = (ld - n) * nrv;
  for (int64_t e = c; e < pad; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / (ld - n), i = n + (e - r * (ld - n));
    out[r * ld + i] = 0.0;
  }
}

__global__ void mask_rows_kernel(float* __restrict__ u, const uint8_t* __restrict__ excl,
                                 int64_t m) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m && excl[i]) u[i] = 0.f;
}

__global__ void zero_pad_kernel(double* __restrict__ v, int64_t n, int64_t ld) {
  const int c = blockIdx.y;
  const int64_t i = n + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ld) v[(int64_t)c * ld + i] = 0.0;
}

inline unsigned g1(int64_t n) { return (unsigned)ceil_div(n, kT); }

}  // namespace

bool one_launch_columns(int64_t n) { return red_blocks(n) <= kClusterRows; }

int red_blocks(int64_t n) {
  int64_t b = ceil_div(n, 4096);
  if (b < 1) b = 1;
  if (b > 256) b = 256;
  return (int)b;
}

// A column kernel on clusters of nb thread blocks, one per column.
template <class... Params, class... Args>
static cudaError_t launch_columns(void (*kernel)(Params...), int nb, int columns, size_t smem,
                                  cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)nb, (unsigned)columns);
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)nb;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = nb > 1 ? 1 : 0;
  count_launches(1);
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t col_dots(const double* a, const double* b, int64_t n, int64_t ld, int q,
                     double* partial, double* out, cudaStream_t st) {
  const int nb = red_blocks(n);
  if (nb <= kClusterRows) {
    return launch_columns(dots_column_kernel, nb, q, 0, st, a, b, q, false, (const double*)nullptr,
                          n, ld, out);
  }
  col_dots_kernel<<<dim3(nb, q), kT, 0, st>>>(a, b, n, ld, partial);
  reduce_partials<<<(unsigned)ceil_div(q, 8), 256, 0, st>>>(partial, nb, q, out);
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t cross_dots(const double* a, int p, const double* b, int q, const double* w, int64_t n,
                       int64_t ld, double* partial, double* out, cudaStream_t st) {
  const int nb = red_blocks(n);
  if (nb <= kClusterRows) {
    return launch_columns(dots_column_kernel, nb, p * q, 0, st, a, b, q, true, w, n, ld, out);
  }
  cross_dots_kernel<<<dim3(nb, p * q), kT, 0, st>>>(a, b, q, w, n, ld, partial);
  reduce_partials<<<(unsigned)ceil_div(p * q, 8), 256, 0, st>>>(partial, nb, p * q, out);
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t pcg_start(const double* b, const double* x0, const double* ax0, const double* d,
                      double* x, double* r, double* z, double* p, int64_t n, int64_t ld, int q,
                      double tol, bool force_step, PcgCols cols, double* partial,
                      double* scratch4q, cudaStream_t st, PcgSeen seen) {
  const int nb = red_blocks(n);
  if (nb <= kClusterRows) {
    return launch_columns(pcg_start_column_kernel, nb, q, 0, st, b, x0, ax0, d, x, r, p, n, ld, tol,
                          force_step ? 1 : 0, cols, seen);
  }
  pcg_start_kernel<<<dim3(nb, q), kT, 0, st>>>(b, x0, ax0, d, x, r, z, p, n, ld, partial);
  reduce_partials<<<(unsigned)ceil_div(3 * q, 8), 256, 0, st>>>(partial, nb, 3 * q, scratch4q);
  pcg_start_finish<<<(unsigned)ceil_div(q, 64), 64, 0, st>>>(
      scratch4q, q, tol, force_step ? 1 : 0, cols,
      reinterpret_cast<unsigned int*>(scratch4q + 3 * (size_t)q));
  count_launches(3);
  return cudaGetLastError();
}

cudaError_t pcg_apply(const double* p, const double* kp, const double* wmax, double tau0,
                      double tau1, double* ap, int64_t n, int64_t ld, int q, PcgCols cols,
                      double* partial, cudaStream_t st) {
  const int nb = red_blocks(n);
  pcg_apply_kernel<true><<<dim3(nb, q), kT, 0, st>>>(p, kp, wmax, tau0, tau1, ap, n, ld,
                                                     cols.state, partial);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t pcg_apply_w(const double* p, const double* kp, const double* w, double tau0,
                        double tau1, double* ap, int64_t n, int64_t ld, int q, PcgCols cols,
                        double* partial, cudaStream_t st) {
  const int nb = red_blocks(n);
  pcg_apply_kernel<false><<<dim3(nb, q), kT, 0, st>>>(p, kp, w, tau0, tau1, ap, n, ld,
                                                      cols.state, partial);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t pcg_iteration(double* x, double* r, double* z, double* p, const double* kp, double* ap,
                          bool w_inverse, const double* wv, double tau0, double tau1,
                          const double* d, int64_t n, int64_t ld, int q, int max_iter,
                          PcgCols cols, double* partial, double* scratch4q, cudaStream_t st,
                          double* kx, PcgSeen seen) {
  const int nb = red_blocks(n);
  if (nb <= kClusterRows) {
    auto k = w_inverse ? pcg_iteration_kernel<true> : pcg_iteration_kernel<false>;
    const size_t smem = (size_t)ceil_div(n, nb) * sizeof(double);  // at most 32 KB
    return launch_columns(k, nb, q, smem, st, x, r, p, kp, wv, tau0, tau1, d, n, ld, max_iter, cols,
                          kx, seen);
  }
  cudaError_t e =
      w_inverse ? pcg_apply(p, kp, wv, tau0, tau1, ap, n, ld, q, cols, partial, st)
                : pcg_apply_w(p, kp, wv, tau0, tau1, ap, n, ld, q, cols, partial, st);
  if (e != cudaSuccess) return e;
  return pcg_step(x, r, z, p, ap, d, n, ld, q, max_iter, cols, partial, scratch4q, st, kx, kp);
}

cudaError_t pcg_step(double* x, double* r, double* z, double* p, const double* ap,
                     const double* d, int64_t n, int64_t ld, int q, int max_iter, PcgCols cols,
                     double* partial, double* scratch4q, cudaStream_t st, double* kx,
                     const double* kp) {
  const int nb = red_blocks(n);
  double* sums = partial + (int64_t)nb * q;  // after pcg_apply's
  pcg_update_kernel<<<dim3(nb, q), kT, 0, st>>>(x, r, z, p, ap, d, n, ld, cols, partial, sums, kx,
                                                kp);
  unsigned gx = (unsigned)ceil_div(n, kT);
  if (gx > 1024) gx = 1024;
  pcg_p_kernel<<<dim3(gx, q), kT, 0, st>>>(p, z, n, ld, partial, sums, nb, max_iter, cols,
                                           reinterpret_cast<unsigned int*>(scratch4q +
                                                                           3 * (size_t)q));
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t sigma_diag(const double* w, double tau0, double tau1, double* wmax, double* d,
                       int64_t n, cudaStream_t st, const double* diagk) {
  sigma_diag_kernel<<<g1(n), kT, 0, st>>>(w, tau0, tau1, diagk, wmax, d, n);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t sigma_diag_w(const double* w, double tau0, double tau1, double* d, int64_t n,
                         cudaStream_t st) {
  sigma_diag_w_kernel<<<g1(n), kT, 0, st>>>(w, tau0, tau1, d, n);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t eta_mu(const double* x, int p, const double* alpha, int trait, double* eta, double* mu,
                   int64_t n, int64_t ld, cudaStream_t st) {
  eta_mu_kernel<<<g1(n), kT, 0, st>>>(x, p, alpha, trait, eta, mu, n, ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t work_vectors(const double* y, const double* eta, const double* mu, int trait,
                         double* w, double* ytil, int64_t n, cudaStream_t st) {
  work_vectors_kernel<<<g1(n), kT, 0, st>>>(y, eta, mu, trait, w, ytil, n);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t init_mu(const double* y, int trait, double* mu, double* eta, int64_t n,
                    cudaStream_t st) {
  init_mu_kernel<<<g1(n), kT, 0, st>>>(y, trait, mu, eta, n);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t sub_combo(const double* from, double* y, int q, const double* a, int p,
                      const double* coef, int64_t n, int64_t ld, cudaStream_t st) {
  sub_combo_kernel<<<dim3(g1(ld), q), kT, 0, st>>>(from, y, q, a, p, coef, n, ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t chol_cols(const double* l, int p, double* t, int q, cudaStream_t st) {
  if (p > kCholMax) return cudaErrorInvalidValue;
  CholFactor f{};
  std::copy(l, l + p * p, f.v);
  chol_cols_kernel<<<(unsigned)ceil_div(q, 64), 64, 0, st>>>(f, p, t, q);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t div_w(const double* v, const double* w, double* out, int64_t n, int64_t ld, int q,
                  cudaStream_t st) {
  div_w_kernel<<<dim3(g1(n), q), kT, 0, st>>>(v, w, out, n, ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t keep_cols(const double* a, const double* b, const KeepCols& cols, int k, double* a_out,
                      double* b_out, int slot, int64_t ld, cudaStream_t st) {
  if (k <= 0) return cudaSuccess;
  keep_cols_kernel<<<dim3((unsigned)ceil_div(ld / 2, kT), k), kT, 0, st>>>(a, b, cols, a_out, b_out,
                                                                           slot, ld);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t rademacher_probes_dev(const uint32_t* key, double* out, int64_t n, int64_t ld, int nrv,
                                  cudaStream_t st) {
  Key8 k;
  for (int i = 0; i < 8; ++i) k.w[i] = key[i];
  const int64_t blocks = ceil_div((int64_t)nrv * n, 16);
  const int64_t pad = (ld - n) * nrv;
  const int64_t threads = blocks > pad ? blocks : pad;
  rademacher_kernel<<<(unsigned)ceil_div(threads > 0 ? threads : 1, kT), kT, 0, st>>>(k, n, ld, nrv, out);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t mask_rows_f32(float* u, const uint8_t* excl, int64_t m, cudaStream_t st) {
  mask_rows_kernel<<<g1(m), kT, 0, st>>>(u, excl, m);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t zero_pad(double* v, int64_t n, int64_t ld, int q, cudaStream_t st) {
  if (ld <= n) return cudaSuccess;
  zero_pad_kernel<<<dim3(g1(ld - n), q), kT, 0, st>>>(v, n, ld);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace saige
