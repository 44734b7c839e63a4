// Lexicographic Gauss-Seidel / SOR and the reference's single V-cycle "mg",
// reproduced exactly on the GPU.
//
// The reference sweeps in place in lexicographic order (k, j, i)
// (src/backends/cpu/solvers/relaxation.cpp:167-289, solver.cpp:808-962): a node
// reads its lower neighbours already updated and its upper neighbours not yet.
// All nodes of one hyperplane i+j+k = d depend only on hyperplanes d-1 and d+1,
// so visiting hyperplanes in increasing d (nodes of a hyperplane in parallel)
// performs exactly the reference's updates in a different but equivalent order.
//
// Small grids run the whole solve in one resident block: boundary closures,
// the sweeps, the max|du| reduction and the stopping test stay on chip and no
// block waits on another. Large grids launch one kernel per hyperplane.
#include <cmath>
#include <cstring>

#include "cluster.cuh"
#include "host.h"
#include "solvers.cuh"

namespace pdeb {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// In-block boundary fill (same closure chain as k_fill_boundary).
__device__ void block_fill_boundary(const GridDev& g, double* u, bool dirichlet_last) {
  const long long nxy = (long long)g.nx * g.ny, nyz = (long long)g.ny * g.nz, nxz = (long long)g.nx * g.nz;
  const long long total = 2 * nyz + 2 * nxz + (g.dim == 3 ? 2 * nxy : 0);
  for (long long t = threadIdx.x; t < total; t += blockDim.x) {
    int i, j, k, f;
    long long r = t;
    if (r < 2 * nyz) {
      f = r < nyz ? kLeft : kRight;
      r %= nyz;
      j = int(r % g.ny);
      k = int(r / g.ny);
      i = f == kLeft ? 0 : g.nx - 1;
    } else if ((r -= 2 * nyz) < 2 * nxz) {
      f = r < nxz ? kBottom : kTop;
      r %= nxz;
      i = int(r % g.nx);
      k = int(r / g.nx);
      j = f == kBottom ? 0 : g.ny - 1;
    } else {
      r -= 2 * nxz;
      f = r < nxy ? kFront : kBack;
      r %= nxy;
      i = int(r % g.nx);
      j = int(r / g.nx);
      k = f == kFront ? 0 : g.nz - 1;
    }
    const bool on[6] = {i == 0, i == g.nx - 1, j == 0, j == g.ny - 1, g.dim == 3 && k == 0,
                        g.dim == 3 && k == g.nz - 1};
    int owner = -1;
    for (int q = 0; q < 6; ++q)
      if (on[q]) {
        owner = q;
        break;
      }
    if (owner != f) continue;
    u[((long long)k * g.ny + j) * g.nx + i] = boundary_final(g, u, i, j, k, dirichlet_last);
  }
}

// One node of the reference sweep: rhs = -(f + nonlinear(old)) - (lap);
// upd = rhs/center; SOR: (1-omega)*old + omega*upd (relaxation.cpp:217-276,
// solver.cpp:884-962).
template <class Coef>
__device__ __forceinline__ double lex_update(const GridDev& g, const Coef& cf, const double* __restrict__ f,
                                             double fc, const NonlinDev& nl, double* u, int i, int j, int k,
                                             double omega, double* delta, int* degenerate) {
  const long long id = ((long long)k * g.ny + j) * g.nx + i;
  const Stencil<double> s = cf.template at<double>(g, id);
  if (fabs(s.c) < 1e-12) {
    *degenerate = 1;
    return 0.0;
  }
  const double old_u = u[id];
  const double zp = g.dim == 3 ? u[id + g.sxy] : 0.0, zm = g.dim == 3 ? u[id - g.sxy] : 0.0;
  const double lap = nb_sum<double>(s, u[id + 1], u[id - 1], u[id + g.nx], u[id - g.nx], zp, zm, g.dim);
  const double rhs = -f_plus_nl(f ? f[id] : fc, nl, old_u) - lap;
  const double upd = __ddiv_rn(rhs, s.c);
  const double updated = (1.0 - omega) * old_u + omega * upd;
  u[id] = updated;
  *delta = fmax(*delta, fabs(updated - old_u));
  return updated;
}

// Visit the interior nodes of hyperplane d with stride `step` from `start`.
template <class Fn>
__device__ __forceinline__ void for_hyperplane(const GridDev& g, int d, long long start, long long step, Fn&& fn) {
  if (g.dim == 2) {
    const int jlo = max(1, d - (g.nx - 2)), jhi = min(g.ny - 2, d - 1);
    for (long long t = start; t <= jhi - jlo; t += step) {
      const int j = jlo + int(t);
      fn(d - j, j, 0);
    }
  } else {
    // (j, k) pairs with i = d - j - k in [1, nx-2]
    const int klo = max(1, d - (g.nx - 2) - (g.ny - 2)), khi = min(g.nz - 2, d - 2);
    if (khi < klo) return;
    const long long nk = khi - klo + 1;
    const long long nj = g.ny - 2;
    for (long long t = start; t < nk * nj; t += step) {
      const int k = klo + int(t / nj), j = 1 + int(t % nj);
      const int i = d - j - k;
      if (i >= 1 && i <= g.nx - 2) fn(i, j, k);
    }
  }
}

__device__ __forceinline__ int hyper_lo(const GridDev& g) { return g.dim == 3 ? 3 : 2; }
__device__ __forceinline__ int hyper_hi(const GridDev& g) {
  return g.dim == 3 ? (g.nx - 2) + (g.ny - 2) + (g.nz - 2) : (g.nx - 2) + (g.ny - 2);
}

// Whole GS/SOR solve in one block. Iteration sequence of the reference:
// 2D closures then sweep (relaxation.cpp:134-289); 3D sweep then closures
// (solver.cpp:769-981; the initial closures are applied by the host).
template <class Coef>
__global__ void __launch_bounds__(1024) k_gs_lex_block(GridDev g, Coef cf, const double* __restrict__ f, double fc,
                                                       NonlinDev nl, double* u, double omega, double tol, int max_iter,
                                                       unsigned long long budget_ns, Ctl* ctl) {
  __shared__ double red[32];
  __shared__ int s_stop;
  __shared__ int s_degen;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_stop = 0;
    s_degen = 0;
  }
  __syncthreads();
  const unsigned long long t0 = globaltimer_ns();
  int it = 0, status = PDEB200_ERR_NOT_CONVERGED;
  double delta_out = 0.0;
  for (it = 0; it < max_iter; ++it) {
    if (g.dim == 2) {
      block_fill_boundary(g, u, false);  // Neumann/Robin closures only (relaxation.cpp:135)
      __syncthreads();
    }
    double delta = 0.0;
    int degen = 0;
    const int dlo = hyper_lo(g), dhi = hyper_hi(g);
    for (int d = dlo; d <= dhi; ++d) {
      for_hyperplane(g, d, tid, blockDim.x,
                     [&](int i, int j, int k) { lex_update(g, cf, f, fc, nl, u, i, j, k, omega, &delta, &degen); });
      __syncthreads();
    }
    if (degen) s_degen = 1;
    // block max of delta
    for (int off = 16; off > 0; off >>= 1) delta = fmax(delta, __shfl_down_sync(0xffffffffu, delta, off));
    if ((tid & 31) == 0) red[tid >> 5] = delta;
    __syncthreads();
    if (tid < 32) {
      double v = tid < (int)(blockDim.x + 31) / 32 ? red[tid] : 0.0;
      for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, off));
      if (tid == 0) red[0] = v;
    }
    __syncthreads();
    const double md = red[0];
    if (g.dim == 3) {
      block_fill_boundary(g, u, true);
      __syncthreads();
    }
    delta_out = md;
    if (tid == 0) {
      if (s_degen) s_stop = 2;
      else if (md < tol) s_stop = 1;
      else if (globaltimer_ns() - t0 > budget_ns) s_stop = 3;
    }
    __syncthreads();
    if (s_stop) break;
  }
  if (tid == 0) {
    const int stop = s_stop;
    if (stop == 1) status = PDEB200_OK;
    else if (stop == 2) status = PDEB200_ERR_DEGENERATE;
    else if (stop == 3) status = PDEB200_ERR_TIMEOUT;
    ctl->iter = stop ? it + 1 : it;
    ctl->delta = delta_out;
    ctl->status = status;
    ctl->done = 1;
  }
}

// ------------------------------------------ lexicographic Gauss-Seidel / SOR

constexpr int kLexSweeps = 512;   // sweeps of a batch (tested together)

struct ClusterLexArgs {
  const double* f;
  double f_const, omega, tol;
  int max_iter;
  int buf_nodes, slots;
  double* save;                    // csize * buf_nodes: the field at the start of a batch
  unsigned long long budget_ns;
};

// A Gauss-Seidel / SOR solve in the reference's lexicographic order.
//
// A sweep visits hyperplanes d = i + j (+ k) in order; a node reads
// hyperplane d - 1 of this sweep and d + 1 of the one before. So sweep s can
// work on hyperplane d at step 2 s + d: everything it reads was written one
// step earlier, and all sweeps in flight work at once. In steady state a
// step updates every node of one parity, and a sweep costs two steps instead
// of one barrier per hyperplane; every value is the one of the sequential
// order.
//
// The stopping test needs max|du| of each sweep over steps that overlap with
// the following sweeps'. A batch of sweeps runs to its end with one flag
// per sweep ("some |du| >= tol"). When a sweep of the batch passes, the field
// at the start of the batch is restored and the sweeps before that one are run
// again; the last sweep always runs alone, with its maximum (the
// reported delta) and, in 2D, without the closures that the reference
// applies before a sweep only. Batches grow from 64 to kLexSweeps.
//
// Bound by latency, one barrier and a dependent chain per step: 97x65 with
// Robin and Neumann faces, tol 1e-6, 483 -> 16.5 ms against one barrier per
// hyperplane in one block (k_gs_lex_block).
template <int D, class Coef, bool NL>
__global__ void __launch_bounds__(kClusterThreads + 32) k_cluster_lex(GridDev g, Coef cf, ClusterLexArgs a, NonlinDev nl,
                                                             double* __restrict__ u, Ctl* ctl) {
  extern __shared__ double sm[];
  __shared__ FaceDev face[6];
  __shared__ unsigned fail[kLexSweeps];   // this CTA's flags; CTA 0 gathers the others' in all_fail
  __shared__ unsigned all_fail[kLexSweeps];
  __shared__ double wmax[kClusterThreads / 32];
  __shared__ double cmax[kClusterMax];
  __shared__ unsigned long long mbs[2];
  __shared__ unsigned first_pass, flags;  // flags (CTA 0): 1 degenerate, 2 out of time
  const unsigned csize = cl_size(), rank = cl_rank();
  const Slab s = make_slab(g, rank, csize);
  // all threads copy, the last warp controls the exchange instead of updating nodes
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int nu = nt - 32, nwarps = nu >> 5;
  const bool control = warp == nwarps;
  constexpr bool is3 = D == 3;
  const int half = (g.nx - 1) / 2;              // slots of one parity of a row
  const int H = is3 ? g.ny - 2 : 1;
  const int cnt = s.n * H * half;               // slots of one parity
  double* x = sm;
  double* sf = x + a.buf_nodes;
  uint2* tab = reinterpret_cast<uint2*>(sf + a.slots);  // entry and hyperplane
  double* save = a.save + (size_t)rank * a.buf_nodes;
  const unsigned long long t0 = globaltimer_ns();
  if (tid < 6) face[tid] = g.face[tid];
  if (tid == 0) flags = 0;
  const unsigned closing = cl_closing(g);
  ClusterExchange ex;
  ex.init(s, rank, x, mbs);
  constexpr bool kConstCoef = std::is_same<Coef, CoefConst>::value;
  RoundedDiv div;
  if constexpr (kConstCoef) div.init(cf.c);
  cl_sync(csize);  // flags of CTA 0 cleared before any CTA sets them
  const int local = (s.n + 2) * s.L;
  for (int t = tid; t < local; t += nt) x[t] = u[s.off0 + t];
  for (int t = tid; t < 2 * cnt; t += nt) {
    const int p = t >= cnt, r = t - p * cnt, row = r / half, m = r - row * half;
    const int layer = row / H, q = row - layer * H;
    const int j = is3 ? 1 + q : s.lo + layer, k = is3 ? s.lo + layer : 0;
    const int i = 1 + ((p + j + k + 1) & 1) + 2 * m;
    unsigned e = kClEmpty;
    if (i <= g.nx - 2) {
      e = cl_entry(g, s, i, j, k, closing);
      const int id = s.off0 + (int)((e & kClOffMask) >> 3);
      sf[t] = a.f ? a.f[id] : a.f_const;
      if (fabs(cf.template at<double>(g, (long long)id).c) < 1e-12) cl_store_u32(cl_map(&flags, 0), 1u);
    }
    tab[t] = make_uint2(e, (unsigned)(i + j + k));
  }
  cl_sync(csize);
  const int nx = g.nx, sxy = is3 ? (int)g.sxy : 0;
  const int dlo = is3 ? 3 : 2;
  const int dhi = (g.nx - 2) + (g.ny - 2) + (is3 ? g.nz - 2 : 0);
  // bytes that the neighbours send in a step of parity p: the nodes of that
  // parity in the layers before and after this slab
  unsigned expect[2] = {0u, 0u};
  for (int side = 0; side < 2; ++side) {
    if (side == 0 ? !s.has_prev : !s.has_next) continue;
    const int layer = side == 0 ? s.lo - 1 : s.lo + s.n;
    for (int p = 0; p < 2; ++p)
      for (int q = 0; q < H; ++q) {
        const int i0 = 1 + ((p + layer + (is3 ? 1 + q : 0) + 1) & 1);
        if (i0 <= g.nx - 2) expect[p] += 8u * (unsigned)((g.nx - 2 - i0) / 2 + 1);
      }
  }
  int step = 0;
  // the steps of M sweeps of an aligned field. `close`: face closures after
  // each node; `track`: returns this thread's max|du| (M = 1) instead of
  // setting the sweeps' flags
  auto sweeps = [&](int M, bool close, bool track) -> double {
    double acc = 0.0;
    for (int tau = dlo; tau <= dhi + 2 * (M - 1); ++tau, ++step) {
      const int base = (tau & 1) * cnt;
      const unsigned exp_now = tau & 1 ? expect[1] : expect[0];
      if (control) {
        ex.begin(step, exp_now, lane);
        ex.wait(step);
      } else {
        // kClusterNodes nodes of the parity per trip, all computed before
        // any is stored
        for (int q0 = tid; q0 < cnt; q0 += kClusterNodes * nu) {
          uint2 e[kClusterNodes];
          double rhs[kClusterNodes], old_u[kClusterNodes], upd[kClusterNodes], center[kClusterNodes];
#pragma unroll
          for (int m = 0; m < kClusterNodes; ++m) {
            const int q = base + min(q0 + m * nu, cnt - 1);
            e[m] = tab[q];
            // an empty slot reads its row's neighbourhood and is not stored
            const unsigned off = e[m].x == kClEmpty ? 8u * (unsigned)(s.L + (is3 ? nx : 0) + 1) : e[m].x & kClOffMask;
            const Stencil<double> st = cf.template at<double, D>(g, (long long)s.off0 + (off >> 3));
            const double* c = reinterpret_cast<const double*>(reinterpret_cast<const char*>(x) + off);
            old_u[m] = c[0];
            const double zp = is3 ? c[sxy] : 0.0, zm = is3 ? c[-sxy] : 0.0;
            const double lap = nb_sum<double>(st, c[1], c[-1], c[nx], c[-nx], zp, zm, D);
            const double fv = sf[q];
            rhs[m] = -(NL ? __dadd_rn(fv, nl_eval(nl, old_u[m])) : fv) - lap;
            center[m] = st.c;
          }
          if constexpr (kConstCoef) {
            bool fast = div.safe;
#pragma unroll
            for (int m = 0; m < kClusterNodes; ++m) {
              fast = fast && (e[m].x == kClEmpty || div.in_range(rhs[m]));
              upd[m] = div.fast(rhs[m]);
            }
            if (!fast)
#pragma unroll
              for (int m = 0; m < kClusterNodes; ++m) upd[m] = __ddiv_rn(rhs[m], div.b);
          } else {
#pragma unroll
            for (int m = 0; m < kClusterNodes; ++m) upd[m] = __ddiv_rn(rhs[m], center[m]);
          }
#pragma unroll
          for (int m = 0; m < kClusterNodes; ++m) {
            if (q0 + m * nu >= cnt || e[m].x == kClEmpty) continue;
            const unsigned s2 = (unsigned)(tau - (int)e[m].y);  // twice the sweep of the node
            const bool active = s2 < (unsigned)(2 * M);
            double v = old_u[m];
            if (active) {
              v = (1.0 - a.omega) * old_u[m] + a.omega * upd[m];
              *reinterpret_cast<double*>(reinterpret_cast<char*>(x) + (e[m].x & kClOffMask)) = v;
              const double du = fabs(v - old_u[m]);
              if (track) {
                if (du > acc) acc = du;
              } else if (du >= a.tol) {
                fail[s2 >> 1] = 1u;
              }
            }
            if (e[m].x >> kClFaceShift) {
              const unsigned faces = (e[m].x >> kClFaceShift) & 63u;
              if (active && close && faces) cl_close(g, face, s, x, (int)((e[m].x & kClOffMask) >> 3), faces, v);
              // nodes outside the sweeps' range are sent as they are: the
              // neighbours count every node of the parity
              ex.push(step, e[m].x, 0u, v);
            }
          }
        }
      }
      __syncthreads();
    }
    return acc;
  };
  auto store_own = [&]() {
    for (int t = tid; t < local; t += nt) {
      const int layer = t / s.L;
      if (!((layer == 0 && s.has_prev) || (layer == s.n + 1 && s.has_next))) u[s.off0 + t] = x[t];
    }
  };
  enum { kBatch, kRerun, kLast } phase = kBatch;
  int done = 0, status = PDEB200_ERR_NOT_CONVERGED, batch = 64, M = 0;
  double delta = 0.0;
  const bool degenerate = cl_load_u32(cl_map(&flags, 0)) != 0;
  if (degenerate) {
    status = PDEB200_ERR_DEGENERATE;
    done = 1;
  }
  while (!degenerate) {
    if (phase == kBatch) {
      M = min(batch, a.max_iter - 1 - done);  // the last allowed sweep runs alone
      if (M <= 0) phase = kLast;
    }
    if (phase == kBatch) {
      for (int t = tid; t < local; t += nt) save[t] = x[t];
      for (int t = tid; t < M; t += nt) {
        fail[t] = 0.0 < a.tol ? 0u : 1u;  // max|du| >= 0 never passes a zero tolerance
        all_fail[t] = 0u;
      }
      if (tid == 0) first_pass = (unsigned)M;
      cl_sync(csize);
    } else if (phase == kLast) {
      M = 1;
      if constexpr (!is3) {
        // the closures before the last sweep, edges and corners included: in
        // 2D the reference leaves the boundary like this
        store_own();
        __threadfence();
        cl_sync(csize);
        if (rank == 0) block_fill_boundary(g, u, false);
        __threadfence();
        cl_sync(csize);
        for (int t = tid; t < local; t += nt) x[t] = __ldcg(u + s.off0 + t);
        cl_sync(csize);
      }
    }
    double acc = sweeps(M, phase != kLast || is3, phase == kLast);
    if (phase == kBatch) {
      for (int t = tid; t < M; t += nt)
        if (fail[t]) cl_store_u32(cl_map(&all_fail[t], 0), 1u);
      if (control && lane == 0 && (ex.dead || (rank == 0 && globaltimer_ns() - t0 > a.budget_ns)))
        cl_store_u32(cl_map(&flags, 0), 2u);
      cl_sync(csize);
      for (int t = tid; t < M; t += nt)
        if (!cl_load_u32(cl_map(&all_fail[t], 0))) atomicMin(&first_pass, (unsigned)t);
      const bool late = (cl_load_u32(cl_map(&flags, 0)) & 2u) != 0;
      cl_sync(csize);
      const int pass = (int)first_pass;
      __syncthreads();  // read by all before the next batch sets it
      if (pass < M) {
        for (int t = tid; t < local; t += nt) x[t] = save[t];
        cl_sync(csize);
        M = pass;
        phase = pass > 0 ? kRerun : kLast;
      } else {
        done += M;
        batch = min(2 * batch, kLexSweeps);
        if (late) {
          status = PDEB200_ERR_TIMEOUT;
          break;
        }
      }
    } else if (phase == kRerun) {
      done += M;
      phase = kLast;
      // the last sweep may begin with the parity that this one ended with: the
      // copies of both steps go to the same places, so the first have to be there
      cl_sync(csize);
    } else {
      acc = warp_max_nonneg(acc);
      if (lane == 0 && !control) wmax[warp] = acc;
      __syncthreads();
      if (warp == 0) {
        acc = warp_max_nonneg(lane < nwarps ? wmax[lane] : 0.0);
        if (lane < (int)csize) cl_store(cl_map(&cmax[rank], lane), acc);
      }
      cl_sync(csize);
      for (unsigned c = 0; c < csize; ++c) delta = fmax(delta, cmax[c]);
      ++done;
      if (delta < a.tol) status = PDEB200_OK;
      break;
    }
  }
  store_own();
  if (control && lane == 0 && ex.dead) cl_store_u32(cl_map(&flags, 0), 2u);
  cl_sync(csize);
  if (rank == 0 && tid == 0) {
    if (flags & 2u) status = PDEB200_ERR_TIMEOUT;
    ctl->iter = done;
    ctl->delta = delta;
    ctl->status = status;
    ctl->done = 1;
  }
  cl_sync(csize);  // no CTA leaves while another may still access its shared memory
}

// Multi-block form: one launch per hyperplane; max|du| through an atomic max
// on the (non-negative) double's bit pattern in ctl->aux[0].
template <class Coef>
__global__ void k_gs_lex_plane(GridDev g, Coef cf, const double* __restrict__ f, double fc, NonlinDev nl, double* u,
                               double omega, int d, Ctl* ctl, int* degenerate) {
  if (ctl_stopped(ctl)) return;
  double delta = 0.0;
  int degen = 0;
  for_hyperplane(g, d, gtid(), gstride(),
                 [&](int i, int j, int k) { lex_update(g, cf, f, fc, nl, u, i, j, k, omega, &delta, &degen); });
  if (degen) *degenerate = 1;
  for (int off = 16; off > 0; off >>= 1) delta = fmax(delta, __shfl_down_sync(0xffffffffu, delta, off));
  if ((threadIdx.x & 31) == 0 && delta > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(&ctl->aux[0]), (unsigned long long)__double_as_longlong(delta));
}

// end of a multi-block sweep: stopping test of the reference
__global__ void k_gs_lex_check(Ctl* ctl, double tol) {
  if (ctl_stopped(ctl)) return;
  const double md = ctl->aux[0];
  ctl->delta = md;
  ctl->iter += 1;
  ctl->aux[0] = 0.0;
  if (md < tol) {
    ctl->stop = 1;
    ctl->status = PDEB200_OK;
  } else if (ctl->iter >= ctl->max_iter) {
    ctl->stop = 1;
    ctl->status = PDEB200_ERR_NOT_CONVERGED;
  }
}

template <class Coef>
pdeb200_status gauss_seidel(Context* ctx, DevProblem& P, const Coef& cf, const pdeb200_options* o, double* d_out,
                            pdeb200_report* rep) {
  const GridDev& g = P.g;
  const double omega = o->method == PDEB200_SOR ? o->sor_omega : 1.0;
  if (o->method == PDEB200_SOR && (omega <= 0.0 || omega >= 2.0))
    throw StatusFailure{PDEB200_ERR_INVALID, "SOR omega must be in (0,2)"};
  const int max_iter = o->max_iter > 1 ? o->max_iter : 1;
  PDEB_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double) * g.n, ctx->stream));
  ctl_init(ctx, max_iter, o->tol, 0.0);
  fill_boundary(ctx, g, d_out, nullptr);  // initial closures
  const long long interior = (long long)(g.nx - 2) * (g.ny - 2) * (g.dim == 3 ? g.nz - 2 : 1);
  if (o->gs_ordering == PDEB200_ORDER_REDBLACK)
    throw StatusFailure{PDEB200_ERR_UNSUPPORTED, "red-black ordering is offered through the MG forms"};
  const unsigned long long budget = 60ULL * 1000000000ULL;  // device-time guard of the single-launch forms: 60 s
  const ClusterShape cs = cluster_shape(g, 512, ctx->max_cluster);
  const size_t lex_smem = sizeof(double) * (size_t)cs.buf_nodes + (sizeof(double) + sizeof(uint2)) * (size_t)cs.slots;
  // Grids whose slabs fit in the shared memory of a cluster (about 160k nodes
  // in 2D): 97x65 SOR 483 -> 16.5 ms. A sweep alone takes as many steps there as
  // barriers in one block, and a step visits half of a CTA's nodes, so a run of
  // few sweeps stays in one block (ms in one block / cluster: 97x65 with k 0.29 /
  // 0.33 for 2 sweeps, 0.52 / 0.34 for 4; 374x267 with nodal coefficients 8.7 / 11.1
  // for 8, 17.2 / 11.3 for 16; 2353x3 in one CTA 4.2 / 4.7 for 4, 8.2 / 4.7 for 8).
  if (cs.csize > 0 && lex_smem <= kClusterDynSmem && max_iter >= 4 + cs.cnt_max / 512) {
    Buf save(sizeof(double) * (size_t)cs.buf_nodes * cs.csize, ctx->stream);
    ClusterLexArgs a{P.f, P.f_const, omega, o->tol, max_iter, cs.buf_nodes, cs.slots, save.as<double>(), budget};
    auto kern = g.dim == 3 ? (P.nl.n ? k_cluster_lex<3, Coef, true> : k_cluster_lex<3, Coef, false>)
                           : (P.nl.n ? k_cluster_lex<2, Coef, true> : k_cluster_lex<2, Coef, false>);
    launch_cluster(ctx, cs.csize, cs.threads, lex_smem, kern, g, cf, a, P.nl, d_out, ctx->d_ctl);
    ctx->count();
    if (g.dim == 3) fill_boundary(ctx, g, d_out, nullptr);
    const Ctl& c = ctl_poll(ctx);
    if (rep) {
      rep->iterations = c.iter;
      rep->last_delta = c.delta;
      rep->converged = c.status == PDEB200_OK;
    }
    return (pdeb200_status)c.status;
  }
  if (interior <= (1LL << 18)) {
    k_gs_lex_block<Coef><<<1, 1024, 0, ctx->stream>>>(g, cf, P.f, P.f_const, P.nl, d_out, omega, o->tol, max_iter,
                                                      budget,
                                                      ctx->d_ctl);
    ctx->count();
    const Ctl& c = ctl_poll(ctx);
    if (rep) {
      rep->iterations = c.iter;
      rep->last_delta = c.delta;
      rep->converged = c.status == PDEB200_OK;
    }
    return (pdeb200_status)c.status;
  }
  Buf degen(sizeof(int), ctx->stream);
  PDEB_CUDA(cudaMemsetAsync(degen.as<int>(), 0, sizeof(int), ctx->stream));
  int dlo = g.dim == 3 ? 3 : 2;
  int dhi = g.dim == 3 ? (g.nx - 2) + (g.ny - 2) + (g.nz - 2) : (g.nx - 2) + (g.ny - 2);
  auto iterate = [&](int) {
    if (g.dim == 2) fill_boundary(ctx, g, d_out, ctx->d_ctl, false);
    for (int d = dlo; d <= dhi; ++d) {
      k_gs_lex_plane<Coef><<<vec_blocks((long long)(g.ny) * g.nz, ctx), 256, 0, ctx->stream>>>(
          g, cf, P.f, P.f_const, P.nl, d_out, omega, d, ctx->d_ctl, degen.as<int>());
    }
    ctx->count(dhi - dlo + 1);
    if (g.dim == 3) fill_boundary(ctx, g, d_out, ctx->d_ctl);
    k_gs_lex_check<<<1, 1, 0, ctx->stream>>>(ctx->d_ctl, o->tol);
    ctx->count();
  };
  pdeb200_status st = drive(ctx, o, max_iter, iterate, true);
  const Ctl c = ctl_poll(ctx);
  int dg = 0;
  PDEB_CUDA(cudaMemcpy(&dg, degen.as<int>(), sizeof(int), cudaMemcpyDeviceToHost));
  if (dg) return PDEB200_ERR_DEGENERATE;
  if (rep) {
    rep->iterations = c.iter;
    rep->last_delta = c.delta;
    rep->converged = st == PDEB200_OK;
  }
  return st;
}

template pdeb200_status gauss_seidel<CoefConst>(Context*, DevProblem&, const CoefConst&, const pdeb200_options*,
                                                double*, pdeb200_report*);
template pdeb200_status gauss_seidel<CoefDivk<double>>(Context*, DevProblem&, const CoefDivk<double>&,
                                                       const pdeb200_options*, double*, pdeb200_report*);
template pdeb200_status gauss_seidel<CoefNodal>(Context*, DevProblem&, const CoefNodal&, const pdeb200_options*,
                                                double*, pdeb200_report*);

// ------------------------------------------------ reference single V-cycle

// MultigridVcyclePoisson (src/backends/cpu/solvers/multigrid.cpp:121-222):
// 2D, constant a, b, e, lexicographic GS smoother, full weighting on interior
// coarse nodes, bilinear prolongation-add over the whole fine grid, exactly
// one cycle. Each grid is a Level2 on the device.
struct MgRefLevel {
  int nx, ny;
  double ax, by, center;
  double *u, *b, *r;
};

// SmoothGsPoisson (multigrid.cpp:69-94), hyperplane order, one block
__global__ void __launch_bounds__(1024) k_mgref_smooth(MgRefLevel L, int iters) {
  const int tid = threadIdx.x;
  const int nx = L.nx, ny = L.ny;
  for (int it = 0; it < iters; ++it) {
    for (int d = 2; d <= (nx - 2) + (ny - 2); ++d) {
      const int jlo = max(1, d - (nx - 2)), jhi = min(ny - 2, d - 1);
      for (int t = tid; t <= jhi - jlo; t += blockDim.x) {
        const int j = jlo + t, i = d - j;
        const long long id = (long long)j * nx + i;
        const double rhs = L.b[id] - L.ax * (L.u[id - 1] + L.u[id + 1]) - L.by * (L.u[id - nx] + L.u[id + nx]);
        L.u[id] = __ddiv_rn(rhs, L.center);
      }
      __syncthreads();
    }
  }
}

// ResidualPoisson (multigrid.cpp:96-119): r = b - (center*u + ax*(ul+ur) + by*(ud+uu)) inside, 0 on the boundary
__global__ void k_mgref_residual(MgRefLevel L) {
  const long long n = (long long)L.nx * L.ny;
  for (long long t = gtid(); t < n; t += gstride()) {
    const int i = int(t % L.nx), j = int(t / L.nx);
    if (i == 0 || j == 0 || i == L.nx - 1 || j == L.ny - 1) {
      L.r[t] = 0.0;
      continue;
    }
    const double Au = L.center * L.u[t] + L.ax * (L.u[t - 1] + L.u[t + 1]) + L.by * (L.u[t - L.nx] + L.u[t + L.nx]);
    L.r[t] = L.b[t] - Au;
  }
}

// RestrictFullWeighting (multigrid.cpp:14-36): interior coarse nodes, boundary 0
__global__ void k_mgref_restrict(MgRefLevel F, MgRefLevel C) {
  const long long n = (long long)C.nx * C.ny;
  for (long long t = gtid(); t < n; t += gstride()) {
    const int ic = int(t % C.nx), jc = int(t / C.nx);
    if (ic == 0 || jc == 0 || ic == C.nx - 1 || jc == C.ny - 1) {
      C.b[t] = 0.0;
      C.u[t] = 0.0;
      continue;
    }
    const int ifx = 2 * ic, jf = 2 * jc, fx = F.nx;
    const double* fr = F.r;
    const double c = fr[(long long)jf * fx + ifx] * 0.25;
    const double e = (fr[(long long)jf * fx + ifx - 1] + fr[(long long)jf * fx + ifx + 1] +
                      fr[(long long)(jf - 1) * fx + ifx] + fr[(long long)(jf + 1) * fx + ifx]) * 0.125;
    const double dd = (fr[(long long)(jf - 1) * fx + ifx - 1] + fr[(long long)(jf - 1) * fx + ifx + 1] +
                       fr[(long long)(jf + 1) * fx + ifx - 1] + fr[(long long)(jf + 1) * fx + ifx + 1]) * 0.0625;
    C.b[t] = c + e + dd;
    C.u[t] = 0.0;
  }
}

// ProlongBilinearAdd (multigrid.cpp:38-67) as a gather: fine node (2ic+a,
// 2jc+b) receives exactly one term, from coarse node (ic,jc).
__global__ void k_mgref_prolong(MgRefLevel C, MgRefLevel F) {
  const long long n = (long long)F.nx * F.ny;
  for (long long t = gtid(); t < n; t += gstride()) {
    const int i = int(t % F.nx), j = int(t / F.nx);
    const int ic = i >> 1, jc = j >> 1;
    if (ic >= C.nx || jc >= C.ny) continue;
    const double* cu = C.u;
    const double vc = cu[(long long)jc * C.nx + ic];
    const bool ox = i & 1, oy = j & 1;
    double add;
    if (!ox && !oy) {
      add = vc;
    } else if (ox && !oy) {
      if (!(ic + 1 < C.nx)) continue;
      add = 0.5 * (vc + cu[(long long)jc * C.nx + ic + 1]);
    } else if (!ox && oy) {
      if (!(jc + 1 < C.ny)) continue;
      add = 0.5 * (vc + cu[(long long)(jc + 1) * C.nx + ic]);
    } else {
      if (!(ic + 1 < C.nx && jc + 1 < C.ny)) continue;
      const double vru = cu[(long long)(jc + 1) * C.nx + ic + 1];
      const double vr = cu[(long long)jc * C.nx + ic + 1];
      const double vu = cu[(long long)(jc + 1) * C.nx + ic];
      add = 0.25 * (vc + vr + vu + vru);
    }
    F.u[t] += add;
  }
}

pdeb200_status mg_vcycle_reference(Context* ctx, DevProblem& P, const pdeb200_problem* hp, const pdeb200_options* o,
                                   double* d_out, pdeb200_report* rep) {
  const GridDev& g = P.g;
  if (g.dim != 2 || P.coef_kind != kConst || std::fabs(P.c) > 1e-12 || std::fabs(P.d) > 1e-12)
    throw StatusFailure{PDEB200_ERR_UNSUPPORTED, "Multigrid requires no convection, mixed, or higher-order derivatives"};
  for (int f = 0; f < 4; ++f)
    if (g.face[f].kind != kDirichlet)
      throw StatusFailure{PDEB200_ERR_UNSUPPORTED, "Multigrid requires Dirichlet boundaries on all sides"};
  auto can = [](int nx, int ny) { return nx >= 5 && (nx & 1) && ny >= 5 && (ny & 1); };
  if (!can(g.nx, g.ny)) throw StatusFailure{PDEB200_ERR_UNSUPPORTED, "CPU multigrid solver failed"};
  std::vector<MgRefLevel> lv;
  std::vector<Buf> owned;
  auto coeffs = [&](MgRefLevel& L) {
    const double dx = (hp->xmax - hp->xmin) / (double)(L.nx - 1);
    const double dy = (hp->ymax - hp->ymin) / (double)(L.ny - 1);
    L.ax = hp->a / (dx * dx);
    L.by = hp->b / (dy * dy);
    L.center = -2.0 * L.ax - 2.0 * L.by + hp->e;
  };
  MgRefLevel L0{g.nx, g.ny, 0, 0, 0, d_out, nullptr, nullptr};
  owned.emplace_back(sizeof(double) * g.n, ctx->stream);
  L0.b = owned.back().as<double>();
  owned.emplace_back(sizeof(double) * g.n, ctx->stream);
  L0.r = owned.back().as<double>();
  coeffs(L0);
  lv.push_back(L0);
  const int max_levels = o->mg_max_levels;
  while ((int)lv.size() < max_levels) {
    const MgRefLevel& pr = lv.back();
    if (!can(pr.nx, pr.ny)) break;
    const int ncx = (pr.nx + 1) / 2, ncy = (pr.ny + 1) / 2;
    if (ncx < 3 || ncy < 3) break;
    MgRefLevel c{ncx, ncy, 0, 0, 0, nullptr, nullptr, nullptr};
    for (double** p : {&c.u, &c.b, &c.r}) {
      owned.emplace_back(sizeof(double) * ncx * ncy, ctx->stream);
      *p = owned.back().as<double>();
      PDEB_CUDA(cudaMemsetAsync(*p, 0, sizeof(double) * ncx * ncy, ctx->stream));
    }
    coeffs(c);
    lv.push_back(c);
    if (ncx <= 5 || ncy <= 5) break;
  }
  for (auto& L : lv)
    if (std::fabs(L.center) < 1e-12) throw StatusFailure{PDEB200_ERR_DEGENERATE, "CPU multigrid solver failed"};
  // b = BuildRhs2D, u = Dirichlet closure of zero
  build_full_rhs(ctx, P, L0.b);
  PDEB_CUDA(cudaMemsetAsync(d_out, 0, sizeof(double) * g.n, ctx->stream));
  fill_boundary(ctx, g, d_out, nullptr);
  const int L = (int)lv.size();
  const int pre = o->mg_pre_smooth > 0 ? o->mg_pre_smooth : 0;
  const int post = o->mg_post_smooth > 0 ? o->mg_post_smooth : 0;
  const int coarse = o->mg_coarse_iters > 1 ? o->mg_coarse_iters : 1;
  for (int l = 0; l < L - 1; ++l) {
    k_mgref_smooth<<<1, 1024, 0, ctx->stream>>>(lv[l], pre);
    k_mgref_residual<<<vec_blocks((long long)lv[l].nx * lv[l].ny, ctx), 256, 0, ctx->stream>>>(lv[l]);
    k_mgref_restrict<<<vec_blocks((long long)lv[l + 1].nx * lv[l + 1].ny, ctx), 256, 0, ctx->stream>>>(lv[l],
                                                                                                      lv[l + 1]);
    ctx->count(3);
  }
  k_mgref_smooth<<<1, 1024, 0, ctx->stream>>>(lv[L - 1], coarse);
  ctx->count();
  for (int l = L - 2; l >= 0; --l) {
    k_mgref_prolong<<<vec_blocks((long long)lv[l].nx * lv[l].ny, ctx), 256, 0, ctx->stream>>>(lv[l + 1], lv[l]);
    k_mgref_smooth<<<1, 1024, 0, ctx->stream>>>(lv[l], post);
    ctx->count(2);
  }
  if (rep) {
    rep->iterations = 1;
    rep->converged = 1;
  }
  return PDEB200_OK;
}

}  // namespace pdeb
