// The lower levels of a V-cycle inside one thread-block cluster.
//
// On the levels below about 40k nodes a V-cycle's launches (12 per level, 2 to 5
// us each with their gaps) and the single-block tail cost far more than their
// arithmetic. Here the level that fits first and all levels below it live in
// the shared memory of up to 16 CTAs for one launch: field, right-hand side,
// residual and the folded stencil weights. What does not change during a solve
// (weights, the nodes' places) is laid out once per solve as an image of each
// CTA's shared memory (k_cv_image) and copied in by bulk copies that start
// before the preceding kernel has ended. Levels of more than `single` nodes are
// cut into slabs of layers over the CTAs, with the exchange of cluster.cuh;
// smaller ones run on the first CTA alone. Transfers read the other level's
// slabs in place (distributed shared memory).
//
// Arithmetic: that of the per-level kernels up to rounding, with three
// differences that are exact in exact arithmetic. The smoother multiplies by
// the reciprocal of the folded centre. The residual is evaluated at the first
// colour only: the second colour's was made zero by the pass before. The
// coarsest level's red-black sweeps from zero are a fixed linear map of its
// right-hand side, computed once per solve (k_coarse_map) and applied as one
// small matrix. Transfer weights, boundary extension and its transpose
// included (both are products of per-axis factors), come from tables made on the
// host.
#pragma once

#include <cmath>
#include <cstdlib>
#include <vector>

#include "cluster.cuh"

namespace pdeb {

constexpr int kCvThreads = 512;      // that update nodes; one more warp controls
constexpr int kCvMaxLevels = 10;
constexpr int kCvMaxCoarse = 64;     // interior nodes of the coarsest level
constexpr size_t kCvSmem = kClusterSmem - 2 * 1024;

// restriction onto a coarse index: weights of fine indices i0 .. i0 + 3 (0 outside the interior)
struct RestrictTap {
  double w[4];
  int i0, pad;
};
// prolongation to a fine index: weights and (interior) coarse indices
struct ProlongTap {
  double w[2];
  int i[2];
};

// Sizes and places of one level in the cluster (the same in every CTA). The
// slots of a slab are its nodes by parity, rows padded to an even length; 32
// slots form a block of kCvRows rows of 32 values (1/centre, xm, xp, ym, yp, zm,
// zp, right-hand side), so that a slot's values are constant offsets apart.
struct CvGeo {
  int nx, ny, nz, dim;
  int L, half, H;         // nodes of a layer, slots of one parity of a row, rows of a layer
  int csize;              // CTAs that share the level: 1 or the whole cluster
  int nmax;               // layers of the largest slab
  int nested;             // the pair with the next coarser level is nested 2:1 in every dimension
  unsigned x, r, w, tab;  // byte offsets in shared memory
  float inv_nx, inv_L;
  double lo[3], hi[3];    // this level's boundary extension factors (ExtCoef)
  const RestrictTap* rt[3];  // onto this level from the finer one (levels > 0)
  const ProlongTap* pt[3];   // to this level from the coarser one (levels above the coarsest)
};
constexpr int kCvRows = 8;

// quotient of small non-negative integers (a < 2^20) by the d of inv = 1/d
__device__ __forceinline__ int cv_div(int a, float inv) { return __float2int_rd((float(a) + 0.5f) * inv); }

// A CTA's share of a level.
struct CvMine {
  int lo, n, cnt;      // first layer, layers, slots of one parity
  int nprev;           // layers of the previous CTA (0: none before this one)
  int next;            // a CTA follows
  unsigned expect[2];  // nodes of each parity in the neighbour layers
};

// Layout of the cluster's shared memory: [image: geo, mine, tab and w of every level][x and r].
struct CvLayout {
  size_t image = 0, total = 0;  // bytes
};

template <class Coef, typename T>
struct CvLevel {
  GridDev g;
  Coef cf;
  CvGeo q;
};

template <typename T>
__device__ __forceinline__ T* cl_remote(T* p, unsigned rank) {
  unsigned long long a = (unsigned long long)p, r;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(rank));
  return (T*)r;
}

template <typename T>
__device__ __forceinline__ void cl_put_async(unsigned addr, T v, unsigned mb) {
  if constexpr (sizeof(T) == 8)
    cl_store_async(addr, v, mb);
  else
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_uint(v)), "r"(mb)
                 : "memory");
}

// The slab of CTA `rank` on a level of the cluster.
struct CvSlab {
  int lo, n;  // first layer and number of layers
  __device__ __forceinline__ void init(const CvGeo& q, int rank) {
    const int layers = (q.dim == 3 ? q.nz : q.ny) - 2;
    if (q.csize == 1) {
      lo = 1;
      n = rank == 0 ? layers : 0;
      return;
    }
    const int base = layers / q.csize, rem = layers % q.csize;
    lo = 1 + rank * base + min(rank, rem);
    n = base + (rank < rem ? 1 : 0);
  }
};
// the CTA that owns interior layer `layer`, and the layer's place in its buffers (1 = first owned)
__device__ __forceinline__ void cv_owner(const CvGeo& q, int layer, int& rank, int& place) {
  if (q.csize == 1) {
    rank = 0;
    place = layer;
    return;
  }
  const int layers = (q.dim == 3 ? q.nz : q.ny) - 2;
  const int base = layers / q.csize, rem = layers % q.csize, m = layer - 1, cut = rem * (base + 1);
  if (m < cut) {
    rank = m / (base + 1);
    place = m - rank * (base + 1) + 1;
  } else {
    rank = rem + (m - cut) / base;
    place = (m - cut) % base + 1;
  }
}

// Writes level l of CTA `rank`'s image at `base`: places and folded weights,
// folded(i, j, k) being the folded stencil of an interior node.
template <typename T, class Folded>
__device__ __forceinline__ void cv_write_image(const CvGeo& q, int nlev, int l, int rank, unsigned char* base,
                                               const Folded& folded) {
  CvSlab s;
  s.init(q, rank);
  const bool is3 = q.dim == 3;
  const bool prev = s.lo > 1, next = s.lo + s.n < (is3 ? q.nz : q.ny) - 1;
  const int cnt = s.n * q.H * q.half;
  if (threadIdx.x == 0) {
    reinterpret_cast<CvGeo*>(base)[l] = q;
    CvMine m{s.lo, s.n, cnt, 0, 0, {0u, 0u}};
    if (q.csize > 1 && s.n > 0) {
      CvSlab o;
      o.init(q, rank - 1);
      m.nprev = prev ? o.n : 0;
      m.next = next ? 1 : 0;
      for (int side = 0; side < 2; ++side) {
        if (side == 0 ? !prev : !next) continue;
        const int layer = side == 0 ? s.lo - 1 : s.lo + s.n;
        // nodes of parity p in that layer: rows alternate between the two starts
        const int w0 = (q.nx - 1) / 2, w1 = (q.nx - 2) / 2;  // nodes of a row starting at i = 1, at i = 2
        for (int p = 0; p < 2; ++p) {
          const int first = (p + layer + (is3 ? 1 : 0) + 1) & 1;  // of the first row
          const int rows0 = first == 0 ? (q.H + 1) / 2 : q.H / 2;
          m.expect[p] += (unsigned)(rows0 * w0 + (q.H - rows0) * w1);
        }
      }
    }
    reinterpret_cast<CvMine*>(base + sizeof(CvGeo) * nlev)[l] = m;
  }
  unsigned* tab = reinterpret_cast<unsigned*>(base + q.tab);
  T* w = reinterpret_cast<T*>(base + q.w);
  for (int t = threadIdx.x; t < 2 * cnt; t += blockDim.x) {
    const int p = t >= cnt, u = t - p * cnt, row = u / q.half, m = u - row * q.half;
    const int layer = row / q.H, jj = row - layer * q.H;
    const int j = is3 ? 1 + jj : s.lo + layer, k = is3 ? s.lo + layer : 0;
    const int i = 1 + ((p + j + k + 1) & 1) + 2 * m;
    unsigned e = kClEmpty;
    if (i <= q.nx - 2) {
      e = (unsigned)((layer + 1) * q.L + (is3 ? j * q.nx : 0) + i);
      if (layer == 0 && prev) e |= kClPrev;
      if (layer == s.n - 1 && next) e |= kClNext;
      const Stencil<T> st = folded(i, j, k);
      T* ws = w + (t >> 5) * (32 * kCvRows) + (t & 31);
      ws[0] = T(1) / st.c;
      ws[32] = st.xm;
      ws[64] = st.xp;
      ws[96] = st.ym;
      ws[128] = st.yp;
      ws[160] = st.zm;
      ws[192] = st.zp;
    }
    tab[t] = e;
  }
}

// The image of CTA blockIdx.x, level blockIdx.y.
template <class Coef, typename T>
__global__ void __launch_bounds__(256) k_cv_image(const CvLevel<Coef, T>* __restrict__ lv, int nlev, size_t image,
                                                  unsigned char* __restrict__ out) {
  const int l = blockIdx.y;
  const GridDev& g = lv[l].g;
  cv_write_image<T>(lv[l].q, nlev, l, blockIdx.x, out + (size_t)blockIdx.x * image, [&](int i, int j, int k) {
    Stencil<T> st = lv[l].cf.template at<T>(g, ((long long)k * g.ny + j) * g.nx + i);
    fold_faces<T>(g, i, j, k, st, nullptr);
    return st;
  });
}

// One V-cycle of the image's nlev levels on rhs0, result in x0 (interior and
// zero boundary).
//
// Bound by latency on the small levels (a pass is one barrier, one exchange and
// a dependent chain: 500 to 1300 cycles; on 129x97 and below the SMs issue in 14% of
// their cycles, 18 of 28 stalled warp cycles per issue at the barrier of a pass) and by shared-memory bandwidth on the
// first (16 values of 8 bytes per node: 2100 cycles per pass at 33^3). FP64:
// 33^3 and below 47 us, where the launches and the single-block tail took
// about 172 us; 129x97 and below 38 us (about 170); 51x39x30 and below 42 us (about
// 290, restriction folds included).
//
// NU threads update nodes, 32 more control. go(), called once the preceding
// kernel has completed, tells whether to run. Returns true in one thread of a CTA
// that lost a wait.
template <typename T, int NU, class Go>
__device__ __forceinline__ bool cv_cycle(const unsigned char* __restrict__ image, unsigned image_bytes,
                                         unsigned smem_bytes, int nlev, const T* __restrict__ rhs0,
                                         T* __restrict__ x0, int pre, int post, const double* __restrict__ coarse_map,
                                         int ncoarse, const Go& go) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ unsigned long long mbs[2], mbi;
  __shared__ unsigned image_lost;
  const unsigned csize = cl_size(), rank = cl_rank();
  constexpr int nu = NU;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool control = tid >= nu;
  constexpr unsigned kT = sizeof(T);
  // ---- before the wait for the preceding kernel: what does not depend on it
  if (tid == 0) {
    mb_init(mbs);
    mb_init(mbs + 1);
    mb_init(&mbi);
    mb_init_fence();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mb_expect(&mbi, image_bytes);
    const unsigned char* src = image + (size_t)rank * image_bytes;
    for (unsigned o = 0; o < image_bytes; o += 32768u) {
      const unsigned n = min(32768u, image_bytes - o);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (unsigned)__cvta_generic_to_shared(smem + o)),
                   "l"(src + o), "r"(n), "r"((unsigned)__cvta_generic_to_shared(&mbi))
                   : "memory");
    }
  }
  // fields and residuals zero (boundaries, second-colour residuals)
  for (unsigned o = image_bytes + 16u * tid; o < smem_bytes; o += 16u * blockDim.x)
    *reinterpret_cast<uint4*>(smem + o) = make_uint4(0u, 0u, 0u, 0u);
  const double map0 = coarse_map[0];
  __syncthreads();
  // Without its image a CTA knows no sizes: it touches nothing, and after the
  // first cluster barrier all CTAs leave.
  const bool no_image = __syncthreads_or(!mb_wait(&mbi, 0u)) != 0;
  if (no_image) mb_wait(&mbi, 0u);  // the copies may still be on their way
  if (tid == 0) image_lost = no_image ? 1u : 0u;
  bool dead = false;  // a wait ran out (control warp)
  const CvGeo* geo = reinterpret_cast<const CvGeo*>(smem);
  const CvMine* mine = reinterpret_cast<const CvMine*>(smem + sizeof(CvGeo) * nlev);
  auto X = [&](int l) { return reinterpret_cast<T*>(smem + geo[l].x); };
  auto Rr = [&](int l) { return reinterpret_cast<T*>(smem + geo[l].r); };
  // What a CTA needs of a level while it works on it.
  struct Here {
    int cnt, n, lo, nx, L, my;         // my: distance to the y neighbours (2D: the layers)
    bool is3, dist, work;
    T *x, *w;
    const unsigned* tab;
    unsigned px, nxa, pmb, nmb;        // neighbours' x (shifted for this CTA's offsets) and mbarriers
    unsigned expect[2];                // bytes they send in a pass of each parity
  };
  auto enter = [&](int l) -> Here {
    const CvGeo& q = geo[l];
    const CvMine& m = mine[l];
    Here h;
    h.n = m.n;
    h.lo = m.lo;
    h.cnt = m.cnt;
    h.nx = q.nx;
    h.L = q.L;
    h.is3 = q.dim == 3;
    h.my = h.is3 ? q.nx : q.L;
    h.dist = q.csize > 1;
    h.work = h.dist || rank == 0;
    h.x = X(l);
    h.w = reinterpret_cast<T*>(smem + q.w);
    h.tab = reinterpret_cast<const unsigned*>(smem + q.tab);
    h.px = h.nxa = h.pmb = h.nmb = 0;
    if (m.nprev) {
      h.px = cl_map(h.x, rank - 1) + kT * (unsigned)(m.nprev * q.L);
      h.pmb = cl_map(mbs, rank - 1);
    }
    if (m.next) {
      h.nxa = cl_map(h.x, rank + 1) - kT * (unsigned)(m.n * q.L);
      h.nmb = cl_map(mbs, rank + 1);
    }
    h.expect[0] = kT * m.expect[0];
    h.expect[1] = kT * m.expect[1];
    return h;
  };
  // the values of slot t of a level
  auto slot = [&](const Here& h, int t) -> T* { return h.w + t + (t >> 5) * (32 * (kCvRows - 1)); };
  Here h{};
  if (!no_image) h = enter(0);
  grid_dep_wait();
  grid_dep_release();
  if (!go()) return false;  // the same in every CTA
  if (!no_image) {
    const T* src = rhs0 + (long long)(h.lo - 1) * h.L;
    for (int t = tid; t < 2 * h.cnt; t += blockDim.x) {
      const unsigned e = h.tab[t];
      if (e != kClEmpty) slot(h, t)[7 * 32] = src[e & kClOffMask];
    }
  }
  cl_sync(csize);
  if (__any_sync(0xffffffffu, lane < (int)csize && cl_load_u32(cl_map(&image_lost, lane)) != 0u)) {
    cl_leave(csize);
    return control && lane == 0 && no_image;
  }
  int step = 0;  // exchanges so far (the same in every CTA)
  auto push = [&](unsigned e, T v) {
    const unsigned m = 8u * (unsigned)(step & 1), o = kT * (e & kClOffMask);
    if (e & kClPrev) cl_put_async<T>(h.px + o, v, h.pmb + m);
    if (e & kClNext) cl_put_async<T>(h.nxa + o, v, h.nmb + m);
  };
  // the exchange of one step by the control warp
  auto exchange = [&](unsigned expect) {
    if (lane == 0) mb_expect(mbs + (step & 1), expect);
    if (!dead) dead = !mb_wait(mbs + (step & 1), (unsigned)(step >> 1) & 1u);
  };
  // neighbour sum of a node: c its place in x, ws its slot's values
  auto neighbours = [&](const T* c, const T* ws) -> T {
    T v = ws[64] * c[1] + ws[32] * c[-1] + ws[128] * c[h.my] + ws[96] * c[-h.my];
    if (h.is3) v = v + ws[192] * c[h.L] + ws[160] * c[-h.L];
    return v;
  };
  // one colour pass of the level h; zero: the field is zero (first pass of a sweep from zero)
  auto pass = [&](int color, bool zero) {
    if (h.work) {
      if (control) {
        if (h.dist) exchange(color ? h.expect[1] : h.expect[0]);
      } else {
        const int base = color ? h.cnt : 0;
        for (int t = base + tid; t < base + h.cnt; t += nu) {
          const unsigned e = h.tab[t];
          if (e == kClEmpty) continue;
          T* c = h.x + (e & kClOffMask);
          const T* ws = slot(h, t);
          const T v = (ws[7 * 32] - (zero ? T(0) : neighbours(c, ws))) * ws[0];
          *c = v;
          if (e & (kClPrev | kClNext)) push(e, v);
        }
      }
      __syncthreads();
    }
    if (h.dist) ++step;
  };
  // a level's work done by all of its CTAs before another level reads it
  auto meet = [&](int la, int lb) {
    if (geo[la].csize > 1 || geo[lb].csize > 1)
      cl_sync(csize);
    else if (rank == 0)
      __syncthreads();
  };
  for (int l = 0; l + 1 < nlev; ++l) {
    for (int p = 0; p < pre; ++p) {
      pass(0, p == 0);
      pass(1, false);
    }
    // residual: of the first colour, or of a zero field
    if (h.work && !control) {
      T* r = Rr(l) - h.L;
      for (int t = tid; t < (pre > 0 ? h.cnt : 2 * h.cnt); t += nu) {
        const unsigned e = h.tab[t];
        if (e == kClEmpty) continue;
        const T* ws = slot(h, t);
        T v = ws[7 * 32];
        if (pre > 0) {
          const T* c = h.x + (e & kClOffMask);
          v = v - (c[0] / ws[0] + neighbours(c, ws));
        }
        r[e & kClOffMask] = v;
      }
    }
    meet(l, l + 1);
    // restriction onto the slabs of the coarser level
    const CvGeo& f = geo[l];
    const CvGeo& q = geo[l + 1];
    h = enter(l + 1);
    if (h.work) {
      const bool is3 = h.is3, nested = f.nested && pre > 0;
      for (int t = tid; t < 2 * h.cnt; t += blockDim.x) {
        const unsigned e = h.tab[t];
        if (e == kClEmpty) continue;
        const int off = (int)(e & kClOffMask), layer = cv_div(off, q.inv_L), in = off - layer * q.L;
        const int row = is3 ? cv_div(in, q.inv_nx) : 0;
        const int J = is3 ? row : h.lo + layer - 1, I = is3 ? in - row * q.nx : in, K = is3 ? h.lo + layer - 1 : 0;
        // weights of fine layer kf (2D: row) of this node's column, 0 outside the level
        auto place = [&](int lf) -> const T* {
          int o, pl;
          cv_owner(f, lf, o, pl);
          return cl_remote(Rr(l), (unsigned)o) + (pl - 1) * f.L;
        };
        double acc = 0.0;
        if (nested) {
          // taps 2I - 1 .. 2I + 1; only the first colour's residuals are not zero
          const RestrictTap& ax = q.rt[0][I];
          const RestrictTap& ay = q.rt[1][J];
          const double x0w = ax.w[0], x1w = ax.w[1], x2w = ax.w[2];
          const double y0w = ay.w[0], y1w = ay.w[1], y2w = ay.w[2];
          if (is3) {
            const RestrictTap& az = q.rt[2][K];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
              const T* p = place(2 * K - 1 + cc) + (2 * J - 1) * f.nx + 2 * I - 1;
              const T *p1 = p + f.nx, *p2 = p1 + f.nx;
              double v;
              if (cc == 1)
                v = y0w * (x0w * double(p[0]) + x2w * double(p[2])) + y1w * (x1w * double(p1[1])) +
                    y2w * (x0w * double(p2[0]) + x2w * double(p2[2]));
              else
                v = y0w * (x1w * double(p[1])) + y1w * (x0w * double(p1[0]) + x2w * double(p1[2])) +
                    y2w * (x1w * double(p2[1]));
              acc += az.w[cc] * v;
            }
          } else {
            const T *p = place(2 * J - 1) + 2 * I - 1, *p1 = place(2 * J) + 2 * I - 1, *p2 = place(2 * J + 1) + 2 * I - 1;
            acc = y0w * (x0w * double(p[0]) + x2w * double(p[2])) + y1w * (x1w * double(p1[1])) +
                  y2w * (x0w * double(p2[0]) + x2w * double(p2[2]));
          }
        } else {
          const RestrictTap tx = q.rt[0][I], ty = q.rt[1][J];
          // a row's part: with a first-colour residual only, every other tap is zero
          auto row_sum = [&](const T* p, int parity) -> double {
            if (pre > 0) {
              const double wa = parity ? tx.w[1] : tx.w[0], wb = parity ? tx.w[3] : tx.w[2];
              p += tx.i0 + parity;
              return wa * double(p[0]) + (wb != 0.0 ? wb * double(p[2]) : 0.0);
            }
            double rs = 0.0;
#pragma unroll
            for (int aa = 0; aa < 4; ++aa)
              if (tx.w[aa] != 0.0) rs += tx.w[aa] * double(p[tx.i0 + aa]);
            return rs;
          };
          if (is3) {
            const RestrictTap tz = q.rt[2][K];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
              if (tz.w[cc] == 0.0) continue;
              const T* plane = place(tz.i0 + cc) + ty.i0 * f.nx;
              double sum = 0.0;
#pragma unroll
              for (int bb = 0; bb < 4; ++bb)
                if (ty.w[bb] != 0.0) sum += ty.w[bb] * row_sum(plane + bb * f.nx, (tx.i0 + ty.i0 + bb + tz.i0 + cc) & 1);
              acc += tz.w[cc] * sum;
            }
          } else {
#pragma unroll
            for (int bb = 0; bb < 4; ++bb)
              if (ty.w[bb] != 0.0) acc += ty.w[bb] * row_sum(place(ty.i0 + bb), (tx.i0 + ty.i0 + bb) & 1);
          }
        }
        slot(h, t)[7 * 32] = T(acc);
      }
      __syncthreads();
    }
  }
  // coarsest level: one product with the sweeps' matrix, on the first CTA
  if (rank == 0 && ncoarse == 1) {
    for (int t = tid; t < 2 * h.cnt; t += blockDim.x)
      if (h.tab[t] != kClEmpty) h.x[h.tab[t] & kClOffMask] = T(map0 * double(slot(h, t)[7 * 32]));
  } else if (rank == 0) {
    const CvGeo& q = geo[nlev - 1];
    const int ni = q.nx - 2, nj = q.ny - 2;
    // row-major index of an entry among the interior nodes (the map's order)
    auto index = [&](unsigned e) {
      const int off = (int)(e & kClOffMask), layer = off / q.L, in = off - layer * q.L;
      if (q.dim == 3) return ((layer - 1) * nj + in / q.nx - 1) * ni + in % q.nx - 1;
      return (layer - 1) * ni + in - 1;
    };
    for (int t = tid; t < 2 * h.cnt; t += blockDim.x) {
      if (h.tab[t] == kClEmpty) continue;
      const int row = index(h.tab[t]);
      double acc = 0.0;
      for (int u = 0; u < 2 * h.cnt; ++u)
        if (h.tab[u] != kClEmpty) acc += coarse_map[index(h.tab[u]) * ncoarse + row] * double(slot(h, u)[7 * 32]);
      h.x[h.tab[t] & kClOffMask] = T(acc);
    }
  }
  // up: add the interpolated correction, smooth with the colours reversed
  for (int l = nlev - 2; l >= 0; --l) {
    meet(l + 1, l);
    h = enter(l);
    const CvGeo& q = geo[l];
    const CvGeo& c = geo[l + 1];
    const bool is3 = h.is3;
    if (h.work) {
      // the coarse layers around this slab, boundary extension applied (in FP64: in
      // FP32 its factors' products would be rounded), in the residual's place (free
      // by now) where they fit there. FP32 levels: 65^3 1.855 -> 1.875 ms per mixed
      // solve against products rounded to FP32; applying the factors as the layers
      // are read 1.92, no staging 1.95.
      double* stage = reinterpret_cast<double*>(Rr(l));
      const int first = h.lo >> 1, layers = ((h.lo + h.n) >> 1) - first + 1;  // nested: coarse layers first ..
      const bool staged = q.nested && layers * c.L * sizeof(double) <= q.nmax * q.L * sizeof(T) && h.n > 0;
      if (staged) {
        for (int t = tid; t < layers * c.L; t += blockDim.x) {
          const int ly = cv_div(t, c.inv_L), in = t - ly * c.L, row = is3 ? cv_div(in, c.inv_nx) : 0;
          const int I = in - row * c.nx, S = first + ly;  // S: coarse layer
          const int nl = is3 ? c.nz : c.ny, la = is3 ? 2 : 1;
          double a = S == 0 ? c.lo[la] : (S == nl - 1 ? c.hi[la] : 1.0);
          if (is3) a *= row == 0 ? c.lo[1] : (row == c.ny - 1 ? c.hi[1] : 1.0);
          a *= I == 0 ? c.lo[0] : (I == c.nx - 1 ? c.hi[0] : 1.0);
          int o, pl;
          cv_owner(c, ext_clamp(S, nl), o, pl);
          const T* src = cl_remote(X(l + 1), (unsigned)o) + pl * c.L + (is3 ? ext_clamp(row, c.ny) * c.nx : 0) +
                         ext_clamp(I, c.nx);
          stage[t] = ext_scale(a, double(*src));
        }
        __syncthreads();
      }
      // The first colour is sent to the neighbours, for the second colour's pass,
      // which sends the second colour itself: a copy of it now would go to the
      // same places with nothing to order the two. Without a pass to come none is
      // sent.
      if (control) {
        if (h.dist && post > 0) exchange(h.expect[0]);
      } else {
        for (int t = tid; t < 2 * h.cnt; t += nu) {
          const unsigned e = h.tab[t];
          if (e == kClEmpty) continue;
          const int off = (int)(e & kClOffMask), layer = cv_div(off, q.inv_L), in = off - layer * q.L;
          const int row = is3 ? cv_div(in, q.inv_nx) : 0;
          const int i = in - row * q.nx, s = h.lo + layer - 1;  // s: fine layer
          double v;
          if (staged) {
            // mean of the two coarse nodes around the node on each axis (the same one twice on it)
            const double* a0 = stage + ((s >> 1) - first) * c.L + (i >> 1);
            const double* a1 = stage + (((s + 1) >> 1) - first) * c.L + (i >> 1);
            const int d = i & 1;
            if (is3) {
              const int r0 = (row >> 1) * c.nx, r1 = ((row + 1) >> 1) * c.nx;
              v = 0.125 * (((a0[r0] + a0[r0 + d]) + (a0[r1] + a0[r1 + d])) +
                           ((a1[r0] + a1[r0 + d]) + (a1[r1] + a1[r1 + d])));
            } else {
              v = 0.25 * ((a0[0] + a0[d]) + (a1[0] + a1[d]));
            }
          } else {
            const int j = is3 ? row : s;
            const ProlongTap tx = q.pt[0][i], ty = q.pt[1][j];
            v = 0.0;
            for (int cc = 0; cc < (is3 ? 2 : 1); ++cc) {
              double wz = 1.0;
              const T* plane = nullptr;
              int o, pl;
              if (is3) {
                const ProlongTap& tz = q.pt[2][s];
                wz = tz.w[cc];
                if (wz == 0.0) continue;
                cv_owner(c, tz.i[cc], o, pl);
                plane = cl_remote(X(l + 1), (unsigned)o) + pl * c.L;
              }
              double sum = 0.0;
#pragma unroll
              for (int bb = 0; bb < 2; ++bb) {
                if (ty.w[bb] == 0.0) continue;
                const T* p;
                if (is3) {
                  p = plane + ty.i[bb] * c.nx;
                } else {
                  cv_owner(c, ty.i[bb], o, pl);
                  p = cl_remote(X(l + 1), (unsigned)o) + pl * c.L;
                }
                double rs = ext_scale(tx.w[0], double(p[tx.i[0]]));
                if (tx.w[1] != 0.0) rs += tx.w[1] * double(p[tx.i[1]]);
                sum += ty.w[bb] * rs;
              }
              v += wz * sum;
            }
          }
          const T nv = T(double(h.x[off]) + v);
          h.x[off] = nv;
          if (post > 0 && t < h.cnt && (e & (kClPrev | kClNext))) push(e, nv);
        }
      }
      __syncthreads();
    }
    if (h.dist && post > 0) ++step;
    for (int p = 0; p < post; ++p) {
      pass(1, false);
      pass(0, false);
    }
  }
  __syncthreads();
  for (int t = tid; t < h.n * h.L; t += blockDim.x) x0[(long long)h.lo * h.L + t] = h.x[h.L + t];
  cl_leave(csize);
  return control && lane == 0 && dead;
}

template <typename T>
__global__ void __launch_bounds__(kCvThreads + 32) k_cluster_vcycle(const unsigned char* __restrict__ image,
                                                                    unsigned image_bytes, unsigned smem_bytes, int nlev,
                                                                    const T* __restrict__ rhs0, T* __restrict__ x0,
                                                                    int pre, int post,
                                                                    const double* __restrict__ coarse_map, int ncoarse,
                                                                    Ctl* ctl) {
  // the flag is not written while this kernel runs
  if (cv_cycle<T, kCvThreads>(image, image_bytes, smem_bytes, nlev, rhs0, x0, pre, post, coarse_map, ncoarse,
                              [&]() { return !ctl_skip(ctl); })) {
    ctl->status = PDEB200_ERR_TIMEOUT;
    ctl->done = 1;
  }
}

// Column `col` of the coarsest level's map: `sweeps` red-black sweeps from
// zero for the unit right-hand side, in FP64 (map[col * n + row], interior nodes
// in row-major order). folded(i, j, k) as in cv_write_image. One block of
// kCvMaxCoarse threads.
template <class Folded>
__device__ __forceinline__ void cv_map_column(const GridDev& g, int sweeps, int col, double* __restrict__ map,
                                              const Folded& folded) {
  __shared__ double sx[kCvMaxCoarse];
  const int ni = g.nx - 2, nj = g.ny - 2, nk = g.dim == 3 ? g.nz - 2 : 1, n = ni * nj * nk;
  const int t = threadIdx.x;
  const int i = t % ni, j = (t / ni) % nj, k = t / (ni * nj);
  Stencil<double> s{};
  if (t < n) s = folded(i + 1, j + 1, g.dim == 3 ? k + 1 : 0);
  sx[t] = 0.0;
  __syncthreads();
  if (n == 1) sweeps = 1;  // the first sweep is the fixed point
  for (int q = 0; q < 2 * sweeps; ++q) {
    // colour of node (i + 1, j + 1, k + 1): the parity of its coordinates' sum
    const int par = (i + j + 2 + (g.dim == 3 ? k + 1 : 0)) & 1;
    if (t < n && par == (q & 1)) {
      double v = t == col ? 1.0 : 0.0;
      if (i > 0) v -= s.xm * sx[t - 1];
      if (i < ni - 1) v -= s.xp * sx[t + 1];
      if (j > 0) v -= s.ym * sx[t - ni];
      if (j < nj - 1) v -= s.yp * sx[t + ni];
      if (k > 0) v -= s.zm * sx[t - ni * nj];
      if (k < nk - 1) v -= s.zp * sx[t + ni * nj];
      sx[t] = v / s.c;
    }
    __syncthreads();
  }
  if (t < n) map[col * n + t] = sx[t];
}

template <class Coef>
__global__ void __launch_bounds__(kCvMaxCoarse) k_coarse_map(GridDev g, Coef cf, int sweeps, double* __restrict__ map) {
  cv_map_column(g, sweeps, blockIdx.x, map, [&](int i, int j, int k) {
    Stencil<double> s = cf.template at<double>(g, ((long long)k * g.ny + j) * g.nx + i);
    fold_faces<double>(g, i, j, k, s, nullptr);
    return s;
  });
}

// Restriction of one level pair as a launch: full weighting and the transpose
// of the boundary extension in one pass over the interior coarse nodes (the
// extension's transpose is in the taps of the nodes next to a face, so no
// second launch gathers boundary nodes). A thread owns a coarse column and
// marches in z; nested 2:1 in z the fine plane between two coarse planes is
// summed once, else the sums of a window of four fine planes are kept.
// Against full weighting at every node plus the gathering launch: the three
// largest pairs of a 257^3 V-cycle 98 -> 48 us, a 100x77x58 pair 14.3 -> 4.9 us.
template <typename T>
__global__ void __launch_bounds__(kBx* kBy) k_restrict_taps(LevelGeo gf, LevelGeo gc, const RestrictTap* __restrict__ tx,
                                                            const RestrictTap* __restrict__ ty,
                                                            const RestrictTap* __restrict__ tz, int nested_xy,
                                                            int nested_z, const T* __restrict__ rf,
                                                            T* __restrict__ bc, const Ctl* ctl) {
  if (ctl_skip_dep(ctl)) return;
  const int I = 1 + blockIdx.x * kBx + threadIdx.x, J = 1 + blockIdx.y * kBy + threadIdx.y;
  const int kb = gc.dim == 3 ? 1 : 0, ke = gc.dim == 3 ? gc.nz - 1 : 1;
  const int chunk = (ke - kb + gridDim.z - 1) / gridDim.z;
  const int K0 = kb + blockIdx.z * chunk, K1 = min(ke, K0 + chunk);
  if (I > gc.nx - 2 || J > gc.ny - 2 || K0 >= K1) return;
  const RestrictTap ax = tx[I], ay = ty[J];
  const T* base = rf + (long long)ay.i0 * gf.nx + ax.i0;
  auto plane = [&](int kf) -> double {
    const T* p = base + (long long)kf * gf.sxy;
    double acc = 0.0;
    if (nested_xy) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const T* row = p + b * gf.nx;
        acc += ay.w[b] * (ax.w[0] * double(row[0]) + ax.w[1] * double(row[1]) + ax.w[2] * double(row[2]));
      }
    } else {
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        if (ay.w[b] == 0.0) continue;
        const T* row = p + b * gf.nx;
        double rs = 0.0;
#pragma unroll
        for (int a = 0; a < 4; ++a)
          if (ax.w[a] != 0.0) rs += ax.w[a] * double(row[a]);
        acc += ay.w[b] * rs;
      }
    }
    return acc;
  };
  T* out = bc + (long long)K0 * gc.sxy + (long long)J * gc.nx + I;
  if (gc.dim != 3) {
    *out = T(plane(0));
    return;
  }
  if (nested_z) {
    double below = plane(2 * K0 - 1);
#pragma unroll 2
    for (int K = K0; K < K1; ++K, out += gc.sxy) {
      const double mid = plane(2 * K), above = plane(2 * K + 1);
      const RestrictTap& az = tz[K];
      *out = T(az.w[0] * below + az.w[1] * mid + az.w[2] * above);
      below = above;
    }
    return;
  }
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;  // sums of planes at .. at + 3, the first `have` of them
  int at = 0, have = 0;
  for (int K = K0; K < K1; ++K, out += gc.sxy) {
    const RestrictTap& az = tz[K];
    while (have > 0 && at < az.i0) {
      s0 = s1;
      s1 = s2;
      s2 = s3;
      ++at;
      --have;
    }
    if (have == 0) at = az.i0;
    if (have <= 0 && az.w[0] != 0.0) s0 = plane(at);
    if (have <= 1 && az.w[1] != 0.0) s1 = plane(at + 1);
    if (have <= 2 && az.w[2] != 0.0) s2 = plane(at + 2);
    if (have <= 3 && az.w[3] != 0.0) s3 = plane(at + 3);
    have = az.w[0] == 0.0 ? 0 : (az.w[1] == 0.0 ? 1 : (az.w[2] == 0.0 ? 2 : (az.w[3] == 0.0 ? 3 : 4)));
    *out = T(az.w[0] * s0 + az.w[1] * s1 + az.w[2] * s2 + az.w[3] * s3);
  }
}

// taps of coarse index I on one axis: full weighting plus the transpose of the
// boundary extension (lo, hi: the closure factors of the axis's faces), interior fine nodes only
__host__ __device__ inline RestrictTap restrict_tap(int I, int n, int nc, double lo, double hi) {
  RestrictTap t{{0, 0, 0, 0}, 0, 0};
  const int den = n - 1, m = nc - 1;
  auto full = [&](int J, int i) -> double {
    if (nc == n) return i == J ? 1.0 : 0.0;
    long long d = (long long)i * m - (long long)J * den;
    d = d < 0 ? -d : d;
    return d < den ? double(m) / double(den) * (1.0 - double(d) / double(den)) : 0.0;
  };
  // with the boundary indices 0 and nc - 1 folded into I
  auto weight = [&](int i) -> double {
    if (i < 1 || i > n - 2) return 0.0;
    double w = full(I, i);
    if (I == 1) w += lo * full(0, i);
    if (I == nc - 2) w += hi * full(nc - 1, i);
    return w;
  };
  int i0 = nc == n ? I : (int)floor(double(I - 1) * den / m);
  if (i0 < 1) i0 = 1;
  while (i0 < n - 2 && full(I, i0) == 0.0) ++i0;
  t.i0 = i0;
  for (int q = 0; q < 4; ++q) t.w[q] = weight(i0 + q);
  return t;
}

__host__ __device__ inline ProlongTap prolong_tap(int i, int n, int nc, double lo, double hi) {
  ProlongTap t{{1.0, 0.0}, {0, 0}};
  int I0;
  double s;
  if (nc == n) {
    I0 = i;
    s = 0.0;
  } else {
    const long long num = (long long)i * (nc - 1);
    I0 = (int)(num / (n - 1));
    s = double(num - (long long)I0 * (n - 1)) / double(n - 1);
  }
  for (int q = 0; q < 2; ++q) {
    const int I = I0 + q;
    const double a = I == 0 ? lo : (I == nc - 1 ? hi : 1.0);
    t.w[q] = (q ? s : 1.0 - s) * (I <= nc - 1 ? a : 0.0);
    t.i[q] = I < 1 ? 1 : (I > nc - 2 ? nc - 2 : I);
  }
  return t;
}

// ------------------------------------------------------------- host side

// Places the levels q[0 .. n) (grids g) in shared memory; levels of at most
// `single` interior nodes go to the first CTA alone.
template <typename T>
inline CvLayout cv_layout(const GridDev* g, int n, int csize, int single, CvGeo* q) {
  CvLayout y;
  size_t at = ((sizeof(CvGeo) + sizeof(CvMine)) * n + 127) / 128 * 128;
  auto take = [&](size_t bytes) {
    const size_t p = at;
    at += (bytes + 15) / 16 * 16;
    return (unsigned)p;
  };
  for (int l = 0; l < n; ++l) {
    CvGeo& c = q[l];
    c.nx = g[l].nx;
    c.ny = g[l].ny;
    c.nz = g[l].nz;
    c.dim = g[l].dim;
    c.L = c.dim == 3 ? (int)g[l].sxy : c.nx;
    c.half = (c.nx - 1) / 2;
    c.H = c.dim == 3 ? c.ny - 2 : 1;
    c.inv_nx = 1.0f / float(c.nx);
    c.inv_L = 1.0f / float(c.L);
    const int layers = (c.dim == 3 ? c.nz : c.ny) - 2;
    const long long interior = (long long)(c.nx - 2) * c.H * layers;
    c.csize = csize > 1 && interior > single && l + 1 < n ? csize : 1;
    c.nmax = (layers + c.csize - 1) / c.csize;
    c.nested = l + 1 < n && 2 * g[l + 1].nx - 1 == c.nx && 2 * g[l + 1].ny - 1 == c.ny &&
               (c.dim != 3 || 2 * g[l + 1].nz - 1 == c.nz);
    const size_t slots = 2 * (size_t)c.nmax * c.H * c.half;
    c.tab = take(sizeof(unsigned) * slots);
    c.w = take(sizeof(T) * kCvRows * ((slots + 31) / 32 * 32));
  }
  y.image = at;
  for (int l = 0; l < n; ++l) {
    q[l].x = take(sizeof(T) * (size_t)(q[l].nmax + 2) * q[l].L);
    q[l].r = l + 1 < n ? take(sizeof(T) * (size_t)q[l].nmax * q[l].L) : q[l].x;
  }
  y.total = at;
  return y;
}

}  // namespace pdeb
