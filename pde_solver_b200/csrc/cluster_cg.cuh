// Conjugate gradients inside one thread-block cluster: the reference CG on the
// full grid and the pressure projection's CG, for grids whose direction
// vector fits in the shared memory of 16 CTAs.
//
// An iteration of a small grid is about a microsecond of arithmetic behind
// three or four launches (each 2 to 5 us with its reduction). Here the vectors
// stay with the CTAs (slabs of whole layers, boundary layers included) and an
// iteration needs two sums over the cluster. A control warp makes them: it adds
// the warps' parts, sends the block's to every CTA with st.async, waits for
// theirs, adds them in CTA order (the same number in every CTA) and derives the
// scalars. The neighbours' layers of p are not exchanged: each CTA keeps a copy
// of the layer before and after its own and updates it like its own,
// p = r + beta p, from the neighbours' r, which travels while the second sum
// is made.
#pragma once

#include <algorithm>

#include "cluster.cuh"

namespace pdeb {

constexpr int kClusterCgIters = 1024;  // most iterations per launch

constexpr int kCgThreads = 512;  // that update nodes; one more warp controls
constexpr int kCgNodes = 4;       // nodes of a thread in flight at once

enum CgOp { kCgFull = 0, kCgProj2 = 1, kCgProj3 = 2 };

// the projection's operator
struct CgProj {
  double cx, cy, cz, cc;
  int pin;
};

struct ClusterCgArgs {
  double *x, *r, *p, *q;  // q: scratch, used when the vectors stay in global memory
  int iters;              // iterations of this launch
  int nx, ny, nz;
  int relative;           // kCgFull: stop on rr <= tol2 instead of sqrt(rr) < tol
  long long n;
};

struct CgShape {
  int csize, threads;
  bool smem_vectors;  // x, r and q in shared memory too
  size_t smem;
};

// most: Context::max_cluster
inline CgShape cg_shape(int nx, int ny, int nz, int most) {
  const bool is3 = nz > 1;
  const int layers = is3 ? nz : ny;
  const long long L = is3 ? (long long)nx * ny : nx;
  CgShape c{1, 0, false, 0};
  while (2 * c.csize <= most && 2 * c.csize <= layers && L * ((layers + c.csize - 1) / c.csize) > 1024) c.csize *= 2;
  const long long m = (layers + c.csize - 1) / c.csize;
  // p with its halo layers, the neighbours' r layers, a flag byte per node
  const size_t base = sizeof(double) * (size_t)((m + 2) * L + 2 * L) + (size_t)(m * L + 7) / 8 * 8;
  const size_t vec = 3 * sizeof(double) * (size_t)(m * L);
  c.smem_vectors = base + vec <= kClusterDynSmem;
  c.smem = base + (c.smem_vectors ? vec : 0);
  if (c.smem > kClusterDynSmem) c.csize = 0;
  c.threads = kCgThreads + 32;
  return c;
}

// Iterations from r, p, x and the scalars of ctl (left there by the launches
// before the loop), to the stopping test or a.iters. p lies in shared memory;
// SM: so do x, r and q = A p during the launch, else they stay in global memory
// (L2).
// At 256x256 (4096 nodes per CTA) an iteration takes 4.9 us against 19.5 us as
// four launches of a replayed graph: about half of it shared-memory bandwidth
// (33 wavefronts per 32 nodes), 1.2 us the two sums (the SMs issue in 30% of their
// cycles; per issue 4.7 warps wait at barriers, 4.4 for shared memory). Measured slower there:
// 992 threads (5.5 us), x, r, q and p in registers (6.8 us, spills at 8 nodes a
// thread), padded rows with wall cells and an offset table (5.4 us).
template <int OP, class Coef, bool SM>
__global__ void __launch_bounds__(kCgThreads + 32) k_cluster_cg(GridDev g, Coef cf, CgProj pj, ClusterCgArgs a,
                                                                Ctl* ctl) {
  extern __shared__ double sm[];
  __shared__ double part[kCgThreads / 32][3];
  __shared__ double red[2][3][kClusterMax];
  __shared__ unsigned long long mbr[2], mbh;
  __shared__ double s_alpha, s_mean, s_beta;
  __shared__ int s_done;
  if (ctl_skip(ctl)) return;  // the flag does not change while the cluster runs
  const unsigned csize = cl_size(), rank = cl_rank();
  const bool is3 = a.nz > 1;
  const int layers = is3 ? a.nz : a.ny, L = is3 ? a.nx * a.ny : a.nx;
  const int base = layers / (int)csize, rem = layers % (int)csize, nmax = base + (rem ? 1 : 0);
  const int lo = (int)rank * base + min((int)rank, rem), nl = base + ((int)rank < rem ? 1 : 0);
  const bool has_prev = rank > 0, has_next = rank + 1 < csize;
  // the strides are constants: a trip's nodes are immediate offsets apart
  constexpr int nt = kCgThreads, nwarps = nt >> 5;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool control = warp == nwarps;
  const int cnt = nl * L;
  const long long g0 = (long long)lo * L;  // global index of the first owned node
  double* p = sm;                          // owned node t is p[L + t]
  double* rh = p + (nmax + 2) * L;         // r of the layers before and after
  double* vec = rh + 2 * L;
  double* r = SM ? vec : a.r + g0;
  double* x = SM ? vec + nmax * L : a.x + g0;
  double* q = SM ? vec + 2 * nmax * L : a.q + g0;
  // the faces a node lies on
  unsigned char* fl = reinterpret_cast<unsigned char*>(SM ? vec + 3 * nmax * L : vec);
  for (int t = tid; t < cnt; t += blockDim.x) {
    if (SM) {
      r[t] = a.r[g0 + t];
      x[t] = a.x[g0 + t];
    }
    const int layer = t / L, in = t - layer * L;
    const int i = in % a.nx, row = in / a.nx;
    const int j = is3 ? row : lo + layer, k = is3 ? lo + layer : 0;
    fl[t] = (unsigned char)((i == 0 ? 1 : 0) | (i == a.nx - 1 ? 2 : 0) | (j == 0 ? 4 : 0) | (j == a.ny - 1 ? 8 : 0) |
                            (is3 && k == 0 ? 16 : 0) | (is3 && k == a.nz - 1 ? 32 : 0));
  }
  for (int t = tid; t < cnt + 2 * L; t += blockDim.x) {
    const bool in = (t >= L || has_prev) && (t < cnt + L || has_next);
    p[t] = in ? a.p[g0 - L + t] : 0.0;
  }
  if (tid == 0) {
    mb_init(mbr);
    mb_init(mbr + 1);
    mb_init(&mbh);
    mb_init_fence();
    s_done = 0;
  }
  cl_sync(csize);
  // lane c of the control warp sends to CTA c
  const unsigned red_to = lane < (int)csize ? cl_map(&red[0][0][rank], lane) : 0u;
  const unsigned mbr_to = lane < (int)csize ? cl_map(mbr, lane) : 0u;
  // r of this slab's first layer is the previous CTA's "after" layer, of its last one the next CTA's "before" layer
  const unsigned rh_prev = has_prev ? cl_map(rh + L, rank - 1) : 0u, rh_next = has_next ? cl_map(rh, rank + 1) : 0u;
  const unsigned mbh_prev = has_prev ? cl_map(&mbh, rank - 1) : 0u, mbh_next = has_next ? cl_map(&mbh, rank + 1) : 0u;
  const unsigned expect_h = 8u * (unsigned)L * ((has_prev ? 1u : 0u) + (has_next ? 1u : 0u));
  // this thread's first node (of its stride nt) in the last layer
  const int last0 = cnt - L, last_t = last0 + (tid - last0 % nt + nt) % nt;
  bool lost = false;
  // the scalars, carried by every lane of the control warp
  double rz = OP == kCgFull ? ctl->rz : ctl->rr, rr = ctl->rr, rn_last = 0.0;
  const double tol = ctl->tol, tol2 = ctl->tol2, brk = ctl->brk, r0 = ctl->aux[6];
  const int max_iter = ctl->max_iter;
  int iter = ctl->iter, status = 0, flag = 0;
  // the sums of the warps' parts over the cluster, by the control warp after a block barrier
  auto cluster_sum = [&](int which, int it, double (&v)[3], int nv) {
    for (int m = 0; m < nv; ++m) {
      double t = lane < nwarps ? part[lane][m] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      v[m] = t;
    }
    if (lane == 0) mb_expect(mbr + which, 8u * csize * (unsigned)nv);
    __syncwarp();
    if (lane < (int)csize)
      for (int m = 0; m < nv; ++m)
        cl_store_async(red_to + 8u * (unsigned)((which * 3 + m) * kClusterMax), v[m], mbr_to + 8u * (unsigned)which);
    if (!lost) lost = !mb_wait(mbr + which, (unsigned)it & 1u);
    for (int m = 0; m < nv; ++m) {
      double t = lane < (int)csize ? red[which][m][lane] : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      v[m] = __shfl_sync(0xffffffffu, t, 0);
    }
  };
  auto warp_part = [&](int m, double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[warp][m] = v;
  };
  // fn(U, t): the nodes t, t + nt, ..., t + (U - 1) nt of this thread, all of them in range
  auto trips = [&](auto&& fn) {
    int t = tid;
    for (; t + (kCgNodes - 1) * nt < cnt; t += kCgNodes * nt) fn(std::integral_constant<int, kCgNodes>{}, t);
    for (; t < cnt; t += nt) fn(std::integral_constant<int, 1>{}, t);
  };
  for (int it = 0; it < a.iters; ++it) {
    // ---- q = A p, p.q (2D projection: and the sums of q and p for the mean)
    if (!control) {
      double pq = 0.0, sq = 0.0, sp = 0.0;
      trips([&](auto uc, int t0) {
        constexpr int U = decltype(uc)::value;
        double val[U], xc[U];
#pragma unroll
        for (int m = 0; m < U; ++m) {
          const unsigned f = fl[t0 + m * nt];
          const double* c = p + L + t0 + m * nt;
          xc[m] = c[0];
          if constexpr (OP == kCgFull) {
            val[m] = xc[m];
            if (!f) {
              const Stencil<double> s = cf.template at<double>(g, g0 + t0 + m * nt);
              const double zp = is3 ? c[L] : 0.0, zm = is3 ? c[-L] : 0.0;
              val[m] = s.c * xc[m] + nb_sum<double>(s, c[1], c[-1], c[a.nx], c[-a.nx], zp, zm, is3 ? 3 : 2);
            }
          } else {
            // neighbours beyond a wall take the node's own value
            const double xm = f & 1 ? xc[m] : c[-1], xp = f & 2 ? xc[m] : c[1];
            const double ym = f & 4 ? xc[m] : c[-a.nx], yp = f & 8 ? xc[m] : c[a.nx];
            if constexpr (OP == kCgProj2) {
              val[m] = pj.cx * (xp - 2.0 * xc[m] + xm) + pj.cy * (yp - 2.0 * xc[m] + ym);
            } else {
              const double zm = f & 16 ? xc[m] : c[-L], zp = f & 32 ? xc[m] : c[L];
              double lap = pj.cc * xc[m];
              lap += pj.cx * xm;
              lap += pj.cx * xp;
              lap += pj.cy * ym;
              lap += pj.cy * yp;
              lap += pj.cz * zm;
              lap += pj.cz * zp;
              val[m] = pj.pin && g0 + t0 + m * nt == 0 ? xc[m] : lap;
            }
          }
        }
#pragma unroll
        for (int m = 0; m < U; ++m) {
          q[t0 + m * nt] = val[m];
          pq += xc[m] * val[m];
          if constexpr (OP == kCgProj2) {
            sq += val[m];
            sp += xc[m];
          }
        }
      });
      warp_part(0, pq);
      if constexpr (OP == kCgProj2) {
        warp_part(1, sq);
        warp_part(2, sp);
      }
    }
    __syncthreads();
    if (control) {
      double v[3];
      cluster_sum(0, it, v, OP == kCgProj2 ? 3 : 1);
      double pq = v[0], mean = 0.0;
      if constexpr (OP == kCgProj2) {
        mean = v[1] / double(a.n);
        pq -= mean * v[2];
      }
      const bool broke = OP == kCgFull ? (!(fabs(pq) >= brk) || isnan(pq)) : fabs(pq) < brk;
      if (broke) {
        flag = 1;
        status = OP == kCgProj2 ? PDEB200_OK : PDEB200_ERR_BREAKDOWN;
      }
      if (lane == 0) {
        s_alpha = rz / pq;
        s_mean = mean;
        if (broke) s_done = 1;
        if (!broke && expect_h) mb_expect(&mbh, expect_h);
      }
    }
    __syncthreads();
    if (s_done) break;
    // ---- x += alpha p, r -= alpha (q - mean), r.r; the slab's outer layers of r to the neighbours
    if (!control) {
      const double alpha = s_alpha, mean = s_mean;
      double acc = 0.0;
      trips([&](auto uc, int t0) {
        constexpr int U = decltype(uc)::value;
        double xn[U], rn[U];
#pragma unroll
        for (int m = 0; m < U; ++m) {
          const int t = t0 + m * nt;
          xn[m] = x[t] + alpha * p[L + t];
          rn[m] = r[t] - alpha * (OP == kCgProj2 ? q[t] - mean : q[t]);
        }
#pragma unroll
        for (int m = 0; m < U; ++m) {
          x[t0 + m * nt] = xn[m];
          r[t0 + m * nt] = rn[m];
          acc += rn[m] * rn[m];
        }
      });
      if (has_prev)
        for (int t = tid; t < L; t += nt) cl_store_async(rh_prev + 8u * (unsigned)t, r[t], mbh_prev);
      if (has_next)
        for (int t = last_t; t < cnt; t += nt) cl_store_async(rh_next + 8u * (unsigned)(t - last0), r[t], mbh_next);
      warp_part(0, acc);
    }
    __syncthreads();
    if (control) {
      double v[3];
      cluster_sum(1, it, v, 1);
      if (expect_h && !lost) lost = !mb_wait(&mbh, (unsigned)it & 1u);
      const double rnew = v[0];
      iter += 1;
      bool done = false;
      if constexpr (OP == kCgFull) {
        rr = rnew;
        if (a.relative ? rnew <= tol2 : sqrt(rnew) < tol) {
          done = true;
          status = PDEB200_OK;
        } else if (a.relative && isnan(rnew)) {
          done = true;
          status = PDEB200_ERR_BREAKDOWN;
        } else if (iter >= max_iter) {
          done = true;
          status = PDEB200_ERR_NOT_CONVERGED;
        }
        if (lane == 0) s_beta = rnew / rz;
        if (!done) rz = rnew;
      } else {
        const double rn = sqrt(rnew);
        if (rn < tol * r0 || rn < 1e-14) {
          done = true;
          status = PDEB200_OK;
          rn_last = rn;
        } else {
          if (lane == 0) s_beta = rnew / rr;
          rr = rz = rnew;
          if (iter >= max_iter) {
            done = true;
            status = PDEB200_ERR_NOT_CONVERGED;
            rn_last = sqrt(rnew);
          }
        }
      }
      if (done && lane == 0) s_done = 2;
    }
    __syncthreads();
    if (s_done) break;
    // ---- p = r + beta p, the neighbours' layers too
    if (!control) {
      const double beta = s_beta;
      trips([&](auto uc, int t0) {
        constexpr int U = decltype(uc)::value;
        double pn[U];
#pragma unroll
        for (int m = 0; m < U; ++m) pn[m] = r[t0 + m * nt] + beta * p[L + t0 + m * nt];
#pragma unroll
        for (int m = 0; m < U; ++m) p[L + t0 + m * nt] = pn[m];
      });
      if (has_prev)
        for (int t = tid; t < L; t += nt) p[t] = rh[t] + beta * p[t];
      if (has_next)
        for (int t = tid; t < L; t += nt) p[L + cnt + t] = rh[L + t] + beta * p[L + cnt + t];
    }
    __syncthreads();
  }
  __syncthreads();
  for (int t = tid; t < cnt; t += blockDim.x) {
    if (SM) {
      a.x[g0 + t] = x[t];
      a.r[g0 + t] = r[t];
    }
    a.p[g0 + t] = p[L + t];
  }
  if (rank == 0 && control && lane == 0) {
    ctl->iter = iter;
    ctl->rr = rr;
    ctl->rz = rz;
    if (s_done) {
      ctl->status = status;
      ctl->aux[5] = rn_last;
      if (flag && OP != kCgFull) ctl->aux[7] = 1.0;
      ctl->done = 1;
    }
  }
  cl_sync(csize);  // no CTA leaves while another may still write into its shared memory
  if (control && lane == 0 && lost) {
    ctl->status = PDEB200_ERR_TIMEOUT;
    ctl->done = 1;
  }
}

template <int OP, class Coef>
inline auto cluster_cg_kernel(const CgShape& c) {
  return c.smem_vectors ? k_cluster_cg<OP, Coef, true> : k_cluster_cg<OP, Coef, false>;
}

}  // namespace pdeb
