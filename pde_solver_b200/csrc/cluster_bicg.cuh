// The reference BiCGStab in 2D inside one thread-block cluster, bit for bit the
// iteration of the per-step launches.
//
// BiCGStab amplifies roundings: two orders of summation stop at different
// iterations with fields that differ by the tolerance. So the sums here are
// made exactly as grid_reduce makes them: "virtual blocks" of 256 threads with
// the shapes of the launches (256 consecutive nodes for vectors, 32 x 8 nodes for
// stencils), the same trees inside them, their results added in block order
// by the same tree. What is saved is launches: ten per iteration (35 us busy of
// 44 us at 97x81) become five phases between cluster barriers. p, s and x are
// evaluated where they are read (the node and its neighbours, from the vectors
// they are made of) instead of by launches of their own, and t = A s is computed
// before the test of |s|, which leaves x alone when it passes.
#pragma once

#include "cluster.cuh"

namespace pdeb {

constexpr int kBiThreads = 1024;            // four virtual blocks
constexpr int kBiBlocks = 256;              // most virtual blocks (the last tree is one block of 256 threads)
constexpr int kBiRounds = kBiBlocks / (kClusterMax * 4);
constexpr int kBiIters = 1024;              // most iterations per launch

struct ClusterBicgArgs {
  double *x, *x1;                // field and its second buffer
  double *p, *p1, *v, *v1, *r, *s, *t;
  const double *b, *rhat;
  double* partials;              // 2 * 3 * kBiBlocks
  int iters, relative;
};

// The fewest CTAs with one stencil block per virtual block, up to `most`
// (Context::max_cluster); 0: the launches serve the grid
inline int bicg_csize(const GridDev& g, int most) {
  const long long nS = (long long)((g.nx + kBx - 1) / kBx) * ((g.ny + kBy - 1) / kBy);
  if (g.dim != 2 || (g.n + 255) / 256 > kBiBlocks || nS > kBiBlocks) return 0;
  int c = 1;
  while (2 * c <= most && 4 * c < nS) c *= 2;
  return nS <= 4LL * c * kBiRounds ? c : 0;
}

constexpr size_t kBiSmem = sizeof(double) * 5 * kBiThreads * kBiRounds;

// Iterations from x, r, p, v and the scalars of ctl to the stopping test or
// a.iters; the field ends in a.x. Bound by latency: 97x81 with per-node
// coefficients 13 to 20 us per iteration from GPU to GPU (five phases of two L2
// round trips and a releasing cluster barrier; per issue 11.5 warps wait at
// barriers, 3.9 for the fences, 3.8 for L2) against 43 to 62 us as launches; sums in another order (3 phases) would stop at another iteration.
template <class Coef>
__global__ void __launch_bounds__(kBiThreads) k_cluster_bicg(GridDev g, Coef cf, ClusterBicgArgs a, Ctl* ctl) {
  extern __shared__ double wts[];  // folded into rounds: weights c, xp, xm, yp, ym of this thread's nodes
  __shared__ double wsum[4][8][3];
  __shared__ double tot[3];
  __shared__ double fin[8][3];
  if (ctl_skip(ctl)) return;  // the flag does not change while the cluster runs
  const unsigned csize = cl_size(), rank = cl_rank();
  const int tid = threadIdx.x, vt = tid & 255, vb = tid >> 8, vw = vt >> 5, lane = tid & 31;
  const int first = (int)rank * 4 + vb, nvb = (int)csize * 4;
  const int gx = (g.nx + kBx - 1) / kBx, gy = (g.ny + kBy - 1) / kBy;
  const int nS = gx * gy, nV = (int)((g.n + 255) / 256), nx = g.nx, ny = g.ny, n = (int)g.n;
  const int roundsS = (nS + nvb - 1) / nvb, roundsV = (nV + nvb - 1) / nvb;
  // this thread's node of stencil round q: index, or -1; interior: has a stencil
  auto node = [&](int q, bool& interior) -> int {
    const int blk = first + q * nvb;
    interior = false;
    if (blk >= nS) return -1;
    const int i = (blk % gx) * kBx + (vt & 31), j = (blk / gx) * kBy + vw;
    if (i >= nx || j >= ny) return -1;
    interior = i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2;
    return j * nx + i;
  };
  for (int q = 0; q < roundsS; ++q) {
    bool in;
    const int id = node(q, in);
    if (id >= 0 && in) {
      const Stencil<double> st = cf.template at<double, 2>(g, id);
      double* w = wts + q * 5 * kBiThreads + tid;
      w[0] = st.c;
      w[kBiThreads] = st.xp;
      w[2 * kBiThreads] = st.xm;
      w[3 * kBiThreads] = st.yp;
      w[4 * kBiThreads] = st.ym;
    }
  }
  // (A u) at node id of round q from the five values of u
  auto stencil = [&](int q, double c, double xp, double xm, double yp, double ym) -> double {
    const double* w = wts + q * 5 * kBiThreads + tid;
    Stencil<double> st;
    st.c = w[0];
    st.xp = w[kBiThreads];
    st.xm = w[2 * kBiThreads];
    st.yp = w[3 * kBiThreads];
    st.ym = w[4 * kBiThreads];
    st.zp = st.zm = 0.0;
    return st.c * c + nb_sum<double>(st, xp, xm, yp, ym, 0.0, 0.0, 2);
  };
  // the virtual block's sums of acc (block_sum's tree) into the partials of block blk
  // (buffer `buf`; consecutive sums take turns, so none is overwritten before all have read it)
  auto block_part = [&](int buf, int blk, int blocks, double (&acc)[3], int nv) {
    for (int m = 0; m < nv; ++m)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[m] += __shfl_down_sync(0xffffffffu, acc[m], o);
    __syncthreads();
    if (lane == 0)
      for (int m = 0; m < nv; ++m) wsum[vb][vw][m] = acc[m];
    __syncthreads();
    if (vw == 0)
      for (int m = 0; m < nv; ++m) {
        double v = lane < 8 ? wsum[vb][lane][m] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0 && blk < blocks) a.partials[(buf * 3 + m) * kBiBlocks + blk] = v;
      }
  };
  // after the cluster barrier: the partials' sum in every CTA, tot[m]
  auto total = [&](int buf, int blocks, int nv) {
    if (tid < 256)
      for (int m = 0; m < nv; ++m) {
        double v = tid < blocks ? __ldcg(a.partials + (buf * 3 + m) * kBiBlocks + tid) : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) fin[tid >> 5][m] = v;
      }
    __syncthreads();
    if (tid < 32)
      for (int m = 0; m < nv; ++m) {
        double v = lane < 8 ? fin[lane][m] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) tot[m] = v;
      }
    __syncthreads();
  };
  const double tol = ctl->tol, tol2 = ctl->tol2, brk = ctl->brk;
  const int max_iter = ctl->max_iter;
  int iter = ctl->iter, status = 0;
  bool done = false, s_exit = false;
  double rho = ctl->rho, rho_prev = ctl->rho_prev, alpha = ctl->alpha, omega = ctl->omega, rr = ctl->rr;
  double *x = a.x, *xn = a.x1, *p = a.p, *pn = a.p1, *v = a.v, *vn = a.v1;
  cl_sync(csize);
  for (int it = 0; it < a.iters; ++it) {
    // ---- rho = rhat.r
    for (int q = 0; q < roundsV; ++q) {
      const int id = (first + q * nvb) * 256 + vt;
      double acc[3] = {0.0, 0.0, 0.0};
      if (id < n) acc[0] += a.rhat[id] * __ldcg(a.r + id);
      block_part(0, first + q * nvb, nV, acc, 1);
    }
    cl_sync(csize);
    total(0, nV, 1);
    rho = tot[0];
    if (fabs(rho) < brk) {
      done = true;
      status = PDEB200_ERR_BREAKDOWN;
      break;
    }
    const double beta = (rho / rho_prev) * (alpha / omega);
    // ---- p = r + beta (p - omega v), v = A p, rhat.v
    {
      auto pv = [&](int id) -> double { return __ldcg(a.r + id) + beta * (__ldcg(p + id) - omega * __ldcg(v + id)); };
      for (int q = 0; q < roundsS; ++q) {
        bool in;
        const int id = node(q, in);
        double acc[3] = {0.0, 0.0, 0.0};
        if (id >= 0) {
          const double c = pv(id);
          double w = c;
          if (in) w = stencil(q, c, pv(id + 1), pv(id - 1), pv(id + nx), pv(id - nx));
          pn[id] = c;
          vn[id] = w;
          acc[0] += a.rhat[id] * w;
        }
        block_part(1, first + q * nvb, nS, acc, 1);
      }
    }
    cl_sync(csize);
    total(1, nS, 1);
    {
      double* t = p;
      p = pn;
      pn = t;
      t = v;
      v = vn;
      vn = t;
    }
    if (fabs(tot[0]) < brk) {
      done = true;
      status = PDEB200_ERR_BREAKDOWN;
      break;
    }
    alpha = rho / tot[0];
    // ---- s = r - alpha v, t = A s
    {
      auto sv = [&](int id) -> double { return __ldcg(a.r + id) - alpha * __ldcg(v + id); };
      for (int q = 0; q < roundsS; ++q) {
        bool in;
        const int id = node(q, in);
        if (id >= 0) {
          const double c = sv(id);
          double w = c;
          if (in) w = stencil(q, c, sv(id + 1), sv(id - 1), sv(id + nx), sv(id - nx));
          a.s[id] = c;
          a.t[id] = w;
        }
      }
    }
    cl_sync(csize);
    // ---- s.s, t.t, t.s
    for (int q = 0; q < roundsV; ++q) {
      const int id = (first + q * nvb) * 256 + vt;
      double acc[3] = {0.0, 0.0, 0.0};
      if (id < n) {
        const double sv = __ldcg(a.s + id), tv = __ldcg(a.t + id);
        acc[0] += sv * sv;
        acc[1] += tv * tv;
        acc[2] += tv * sv;
      }
      block_part(0, first + q * nvb, nV, acc, 3);
    }
    cl_sync(csize);
    total(0, nV, 3);
    if (a.relative ? tot[0] <= tol2 : sqrt(tot[0]) < tol) {
      done = s_exit = true;
      status = PDEB200_OK;
      iter += 1;
      break;
    }
    if (fabs(tot[1]) < brk) {
      done = true;
      status = PDEB200_ERR_BREAKDOWN;
      break;
    }
    omega = tot[2] / tot[1];
    // ---- x += alpha p + omega s, r = b - A x, r.r
    {
      auto xv = [&](int id) -> double { return __ldcg(x + id) + alpha * __ldcg(p + id) + omega * __ldcg(a.s + id); };
      for (int q = 0; q < roundsS; ++q) {
        bool in;
        const int id = node(q, in);
        double acc[3] = {0.0, 0.0, 0.0};
        if (id >= 0) {
          const double c = xv(id);
          double w = c;
          if (in) w = stencil(q, c, xv(id + 1), xv(id - 1), xv(id + nx), xv(id - nx));
          const double rv = a.b[id] - w;
          xn[id] = c;
          a.r[id] = rv;
          acc[0] += rv * rv;
        }
        block_part(1, first + q * nvb, nS, acc, 1);
      }
    }
    cl_sync(csize);
    total(1, nS, 1);
    {
      double* t = x;
      x = xn;
      xn = t;
    }
    rr = tot[0];
    iter += 1;
    done = true;
    if (a.relative ? rr <= tol2 : sqrt(rr) < tol)
      status = PDEB200_OK;
    else if (fabs(omega) < brk)
      status = PDEB200_ERR_BREAKDOWN;
    else if (iter >= max_iter)
      status = PDEB200_ERR_NOT_CONVERGED;
    else
      done = false;
    if (done) break;
    rho_prev = rho;
  }
  // the field (and, before another launch, p and v) to the first buffers
  const int all = (int)csize * kBiThreads;
  for (int id = (int)rank * kBiThreads + tid; id < n; id += all) {
    const double pv = __ldcg(p + id);
    double xv = __ldcg(x + id);
    if (s_exit) xv = xv + alpha * pv;
    if (x != a.x || s_exit) a.x[id] = xv;
    if (p != a.p) {
      const double vv = __ldcg(v + id);
      a.p[id] = pv;
      a.v[id] = vv;
    }
  }
  if (rank == 0 && tid == 0) {
    ctl->iter = iter;
    ctl->rr = rr;
    ctl->rho = rho;
    ctl->rho_prev = rho_prev;
    ctl->alpha = alpha;
    ctl->omega = omega;
    if (done) {
      ctl->status = status;
      ctl->done = 1;
    }
  }
}

}  // namespace pdeb
