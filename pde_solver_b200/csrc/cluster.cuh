// Whole relaxation runs inside one thread-block cluster.
//
// A Jacobi sweep or a heat step of a small grid is a microsecond of work
// behind two launches, and a lexicographic Gauss-Seidel sweep is one barrier
// per hyperplane. Here up to 16 CTAs of one cluster hold the grid in their
// shared memory and run many sweeps per launch; the CTAs meet in each step by
// their neighbours' copies (ClusterExchange), not by a barrier of all.
//
// The grid is cut into slabs of whole layers along its slowest dimension
// (rows in 2D, planes in 3D). A CTA keeps its layers plus the layer before and
// after them; the thread that updates a node of a slab's first or last layer
// also sends the value to the neighbour CTA's copy (distributed shared
// memory), and the thread that updates a node next to a face writes that
// face's closure, so nothing but the exchange separates two sweeps.
#pragma once

#include "../../include/pdeb200.h"
#include "kernels.cuh"
#include <type_traits>

namespace pdeb {

constexpr int kClusterMax = 16;      // opt-in cluster size (8 is the portable limit)
constexpr int kClusterThreads = 512;  // that update nodes; one more warp controls
constexpr int kClusterNodes = 2;     // nodes of a thread in flight at once
constexpr size_t kClusterSmem = 227 * 1024;
constexpr size_t kClusterDynSmem = kClusterSmem - 10 * 1024;  // the kernels' static shared memory stays below 10 KB

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Barrier of the whole cluster; shared-memory writes before it, remote ones
// included, are visible after it. A single CTA takes the block barrier.
__device__ __forceinline__ void cl_sync(unsigned csize) {
  if (csize == 1) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
// The end of a kernel: no CTA leaves while another may still access its shared
// memory. Nothing is published, so the arrival needs no fence.
__device__ __forceinline__ void cl_leave(unsigned csize) {
  __syncthreads();
  if (csize > 1) {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
// the address of this CTA's shared variable in CTA `rank` of the cluster
__device__ __forceinline__ unsigned cl_map(const void* p, unsigned rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cl_store(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_store_u32(unsigned addr, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned cl_load_u32(unsigned addr) {
  unsigned v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// Exchanges without the cluster barrier. A store of st.async carries the
// number of its bytes to an mbarrier beside its destination, and the receiving
// CTA waits until the bytes of a step are there: about 250 cycles, against 480 to
// 830 cycles for stores ordered by a releasing cluster barrier (256 to 1024
// threads; the barrier alone takes 120 to 180, its fence the rest).
__device__ __forceinline__ void mb_init(unsigned long long* mb) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(mb)) : "memory");
}
__device__ __forceinline__ void mb_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// the one arrival of a phase, with the bytes that complete it
__device__ __forceinline__ void mb_expect(unsigned long long* mb, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(mb)),
               "r"(bytes)
               : "memory");
}
// Waits for a phase of the given parity; false when it did not complete within
// the bound (about a second), which only a lost CTA could cause.
constexpr int kClusterWaitTries = 1 << 20;
__device__ __forceinline__ bool mb_wait(unsigned long long* mb, unsigned parity) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mb);
  for (int t = 0; t < kClusterWaitTries; ++t) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(a), "r"(parity), "r"(1000u)  // at most 1 us per try
        : "memory");
    if (ok) return true;
  }
  return false;
}
// store of v at a cluster address, counted by the mbarrier at cluster address mb
__device__ __forceinline__ void cl_store_async(unsigned addr, double v, unsigned mb) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(mb)
               : "memory");
}

// Warp maximum of non-negative doubles (their bit patterns order as integers).
__device__ __forceinline__ double warp_max_nonneg(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  return __hiloint2double((int)mh, (int)ml);
}

// Correctly rounded quotients by one divisor (the centre of a constant
// stencil, the u_t coefficient): RN(1/b) once, then Markstein's iteration
// (P. Markstein, Computation of elementary functions on the IBM RISC
// System/6000 processor, 1990): with y = RN(1/b) and q within 1 ulp of a/b,
// r = a - b q is exact in one fused multiply-add and RN(q + r y) = RN(a/b). The
// product a y may be 1.5 ulp off, so one step makes q faithful and a second
// one rounds it correctly: five dependent operations instead of the general
// division's 113 cycles. Dividends and divisors outside the range where no
// step underflows or overflows, and a divisor whose significand is all ones
// (the theorem's exception), take the general division; the results are its
// bits (2e10 random pairs compared with it, divisors just below all ones and
// every exponent of the range among them: no difference).
struct RoundedDiv {
  double b, y;
  bool safe;
  __device__ __forceinline__ void init(double d) {
    b = d;
    y = __drcp_rn(d);
    const double m = fabs(d);
    safe = m > 0x1p-200 && m < 0x1p200 && (__double_as_longlong(d) & 0xfffffffffffffLL) != 0xfffffffffffffLL;
  }
  // |a| in [2^-600, 2^600), from its exponent
  __device__ __forceinline__ static bool in_range(double a) {
    return ((unsigned)__double2hiint(a) & 0x7fffffffu) - ((1023u - 600u) << 20) < (1200u << 20);
  }
  // the quotient of a dividend in range by a safe divisor
  __device__ __forceinline__ double fast(double a) const {
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
  }
};

// The slab of one CTA.
struct Slab {
  int L;         // nodes of a layer
  int lo, n;     // first owned layer and their number
  int nprev;     // owned layers of the previous CTA
  int off0;      // global index of local node 0 (layer lo - 1)
  bool has_prev, has_next;
};

__device__ __forceinline__ Slab make_slab(const GridDev& g, int c, int csize) {
  Slab s;
  const int layers = (g.dim == 3 ? g.nz : g.ny) - 2;
  s.L = g.dim == 3 ? (int)g.sxy : g.nx;
  const int base = layers / csize, rem = layers % csize;
  s.lo = 1 + c * base + min(c, rem);
  s.n = base + (c < rem ? 1 : 0);
  s.nprev = base + (c - 1 < rem ? 1 : 0);
  s.off0 = (s.lo - 1) * s.L;
  s.has_prev = c > 0;
  s.has_next = c + 1 < csize;
  return s;
}

// Cluster size and buffer sizes of a grid: the fewest CTAs that leave at most
// `nodes_per_cta` interior nodes to each, up to `most` (Context::max_cluster)
// and one layer each, and
// kClusterNodes nodes per thread. Measured at 129x129 (16 CTAs) per Jacobi
// sweep: 2 nodes per thread 0.90 us, 4 nodes 1.08 us; at 97x65 per SOR solve
// with 512 nodes per CTA 16.5 ms, with 1024 17.9 ms (a step visits half of
// them), with 4 nodes per thread 24.9 ms.
struct ClusterShape {
  int csize;
  int threads;    // with the control warp
  int buf_nodes;  // nodes of the largest slab with the layers around it
  int cnt_max;    // interior nodes of the largest slab
  int slots;      // cnt_max with every row padded to an even length
};

inline ClusterShape cluster_shape(const GridDev& g, int nodes_per_cta, int most) {
  const int layers = (g.dim == 3 ? g.nz : g.ny) - 2;
  const long long L = g.dim == 3 ? g.sxy : g.nx;
  const int rows = g.dim == 3 ? g.ny - 2 : 1;
  const long long WH = (long long)(g.nx - 2) * rows;
  ClusterShape c{1, 0, 0, 0, 0};
  while (2 * c.csize <= most && 2 * c.csize <= layers && WH * ((layers + c.csize - 1) / c.csize) > nodes_per_cta)
    c.csize *= 2;
  const long long n = (layers + c.csize - 1) / c.csize;
  if ((n + 2) * L > kClusterSmem / 8) return ClusterShape{0, 0, 0, 0, 0};
  c.buf_nodes = (int)((n + 2) * L);
  c.cnt_max = (int)(n * WH);
  c.slots = (int)(n * rows * ((g.nx - 1) / 2) * 2);
  c.threads = (c.cnt_max + kClusterNodes - 1) / kClusterNodes;
  c.threads = c.threads >= kClusterThreads ? kClusterThreads : (c.threads + 31) / 32 * 32;
  c.threads += 32;  // the control warp
  return c;
}

// A node's entry: local byte offset, the Neumann and Robin faces it is next to, and
// whether its value is copied to the previous or next CTA. Dirichlet values
// never change: they are in place from the start.
constexpr unsigned kClOffMask = (1u << 20) - 1;  // byte offset in a local buffer
constexpr unsigned kClFaceShift = 20;            // 6 bits
constexpr unsigned kClPrev = 1u << 26, kClNext = 1u << 27;
constexpr unsigned kClEmpty = 0xffffffffu;

__device__ __forceinline__ unsigned cl_entry(const GridDev& g, const Slab& s, int i, int j, int k,
                                             unsigned closing) {
  const int layer = (g.dim == 3 ? k : j) - (s.lo - 1);
  unsigned e = 8u * (unsigned)(layer * s.L + (g.dim == 3 ? j * g.nx : 0) + i);
  unsigned f = (i == 1 ? 1u : 0u) | (i == g.nx - 2 ? 2u : 0u) | (j == 1 ? 4u : 0u) | (j == g.ny - 2 ? 8u : 0u);
  if (g.dim == 3) f |= (k == 1 ? 16u : 0u) | (k == g.nz - 2 ? 32u : 0u);
  e |= (f & closing) << kClFaceShift;
  if (layer == 1 && s.has_prev) e |= kClPrev;
  if (layer == s.n && s.has_next) e |= kClNext;
  return e;
}

// the faces whose closures follow the nodes next to them
__device__ __forceinline__ unsigned cl_closing(const GridDev& g) {
  unsigned m = 0;
  for (int f = 0; f < 6; ++f)
    if (g.face[f].active && g.face[f].kind != kDirichlet) m |= 1u << f;
  return m;
}

// Face closures of the nodes next to node `off`, from its new value v.
__device__ __forceinline__ void cl_close(const GridDev& g, const FaceDev* face, const Slab& s, double* dst, int off,
                                         unsigned faces, double v) {
  while (faces) {
    const int f = __ffs(faces) - 1;
    faces &= faces - 1;
    const FaceDev& F = face[f];
    const int step = f < 2 ? 1 : (f < 4 ? g.nx : s.L);
    int loc = 0;
    if (F.val.a || F.alpha.a || F.beta.a || F.gamma.a) {
      const int id = off + s.off0;
      const int i = id % g.nx, r = id / g.nx;
      const int j = g.dim == 3 ? r % g.ny : r, k = g.dim == 3 ? r / g.ny : 0;
      loc = face_loc(g, f, i, j, k);
    }
    bool ok;
    const double b = closure_value(F, f & 1, loc, v, &ok);
    if (ok) dst[(f & 1) ? off + step : off - step] = b;
  }
}

// Exchange of slab layers with the neighbour CTAs, step by step. A node of the
// first or last layer is copied to the neighbour as it is updated; a CTA goes
// on to the next step when its own threads and its neighbours' copies of this
// step are done. Two mbarriers take turns: a neighbour that is ahead is at most
// one step ahead, since it needs this CTA's copies of a step to begin the one
// after. That also makes its writes safe: a node reads the neighbour's node
// of the same index before its own value, whose copy lets the neighbour go on,
// exists.
struct ClusterExchange {
  unsigned prev, next;        // neighbours' addresses of a buffer's node 0, shifted so that this CTA's offsets apply
  unsigned mb_prev, mb_next;  // the neighbours' mbarriers
  unsigned long long* mb;     // this CTA's two mbarriers
  bool dead;                  // a wait ran out (control warp)

  __device__ __forceinline__ void init(const Slab& s, unsigned rank, const double* buf, unsigned long long* m) {
    mb = m;
    prev = s.has_prev ? cl_map(buf, rank - 1) + 8u * (unsigned)(s.nprev * s.L) : 0u;
    next = s.has_next ? cl_map(buf, rank + 1) - 8u * (unsigned)(s.n * s.L) : 0u;
    mb_prev = s.has_prev ? cl_map(m, rank - 1) : 0u;
    mb_next = s.has_next ? cl_map(m, rank + 1) : 0u;
    dead = false;
    if (threadIdx.x == 0) {
      mb_init(m);
      mb_init(m + 1);
      mb_init_fence();
    }
  }
  // copies of an updated node; bytes: offset of the buffer in use from the one of init()
  __device__ __forceinline__ void push(int step, unsigned e, unsigned bytes, double v) const {
    const unsigned m = 8u * (unsigned)(step & 1), o = bytes + (e & kClOffMask);
    if (e & kClPrev) cl_store_async(prev + o, v, mb_prev + m);
    if (e & kClNext) cl_store_async(next + o, v, mb_next + m);
  }
  // Step numbers count from 0 without gaps. Both are called by the control
  // warp: `expect`: bytes that the neighbours send in this step (possibly none)
  __device__ __forceinline__ void begin(int step, unsigned expect, int lane) {
    if ((mb_prev | mb_next) && lane == 0) mb_expect(mb + (step & 1), expect);
  }
  __device__ __forceinline__ void wait(int step) {
    if ((mb_prev | mb_next) && !dead) dead = !mb_wait(mb + (step & 1), (unsigned)(step >> 1) & 1u);
  }
};

// ------------------------------------------------- Jacobi and forward Euler

struct ClusterSweepArgs {
  const double* f;
  double f_const;
  double tol;              // Jacobi
  int max_iter;            // Jacobi: total sweeps allowed
  double ut, dt;           // heat
  int steps;               // sweeps of this launch
  int buf_nodes;           // local buffer size (nodes)
  int cnt_max;             // most interior nodes of a slab
};

// `steps` sweeps of Jacobi (HEAT false: k_jacobi followed by k_fill_boundary,
// with the reference's stopping test after each sweep) or forward Euler
// (HEAT: k_fe_step followed by k_fill_boundary), the same node arithmetic.
// u is read and written in global memory once per launch.
//
// A control warp beside the warps that update nodes does what is not node work:
// it waits for the neighbours' copies, and it tests a sweep while the next one
// is computed: it combines the warps' maxima of sweep t - 1, sends the block's
// to every CTA, waits for theirs and leaves the verdict for the barrier that
// ends sweep t. Sweep t + 1, which would overwrite the field of sweep t - 1 (two
// buffers), is not begun, so the field returned is the one of the sweep that
// met the tolerance.
//
// Bound by latency: a warp issues one instruction of a node's dependent chain
// about every five cycles (129x129: half of the issue slots of its SMs, of
// 8 resident warps' wait per issue 2.5 on the chain, 1.5 on shared memory, 1.0 at
// the block barrier). 129x129: 0.90 us per sweep in 16 CTAs against
// 7.5 us as two launches in a replayed graph (22392 sweeps 168 -> 20.2 ms); with
// a releasing cluster barrier per sweep and the test in every warp 1.4 us.
template <int D, class Coef, bool HEAT, bool NL>
__global__ void __launch_bounds__(kClusterThreads + 32) k_cluster_sweep(GridDev g, Coef cf, ClusterSweepArgs a,
                                                                   NonlinDev nl, double* __restrict__ u, Ctl* ctl,
                                                                   int* degenerate) {
  extern __shared__ double sm[];
  __shared__ FaceDev face[6];
  __shared__ double wmax[2][kClusterThreads / 32];
  __shared__ double cmax[4][kClusterMax];
  __shared__ unsigned long long mbs[2], mbc[4];
  __shared__ int verdict[2];  // 0 go on, else 1 + status
  if (!HEAT && ctl_stopped(ctl)) return;  // the flag does not change while the cluster runs
  const unsigned csize = cl_size(), rank = cl_rank();
  const Slab s = make_slab(g, rank, csize);
  // the last warp is the control warp
  const int tid = threadIdx.x, nt = blockDim.x - 32, warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
  const bool control = warp == nwarps;
  const int W = g.nx - 2, WH = D == 3 ? W * (g.ny - 2) : W;
  const int cnt = s.n * WH;
  double* sf = sm + 2 * (size_t)a.buf_nodes;
  unsigned* tab = reinterpret_cast<unsigned*>(sf + a.cnt_max);
  if (tid < 6) face[tid] = g.face[tid];
  if (tid < 2) verdict[tid] = 0;
  const unsigned closing = cl_closing(g);
  ClusterExchange ex;
  ex.init(s, rank, sm, mbs);
  if (tid == 0) {
    for (int q = 0; q < 4; ++q) mb_init(mbc + q);
    mb_init_fence();
  }
  const int local = (s.n + 2) * s.L;
  for (int t = tid; t < local; t += blockDim.x) sm[t] = sm[a.buf_nodes + t] = u[s.off0 + t];
  for (int t = tid; t < cnt; t += blockDim.x) {
    const int layer = t / WH, r = t - layer * WH;
    const int i = 1 + r % W, q = r / W;
    const int j = D == 3 ? 1 + q : s.lo + layer, k = D == 3 ? s.lo + layer : 0;
    const unsigned e = cl_entry(g, s, i, j, k, closing);
    tab[t] = e;
    sf[t] = a.f ? a.f[s.off0 + (int)((e & kClOffMask) >> 3)] : a.f_const;
  }
  const int iter0 = HEAT ? 0 : ctl->iter;
  // lane c of the control warp sends the block maximum to CTA c
  const unsigned cmax_to = lane < (int)csize ? cl_map(&cmax[0][rank], lane) : 0u;
  const unsigned mbc_to = lane < (int)csize ? cl_map(mbc, lane) : 0u;
  cl_sync(csize);
  const int nx = g.nx, sxy = D == 3 ? (int)g.sxy : 0;
  const unsigned expect = 8u * (unsigned)WH * ((s.has_prev ? 1u : 0u) + (s.has_next ? 1u : 0u));
  constexpr bool kConstCoef = std::is_same<Coef, CoefConst>::value;
  RoundedDiv div;  // by the constant centre, or by the u_t coefficient
  if constexpr (HEAT)
    div.init(a.ut);
  else if constexpr (kConstCoef)
    div.init(cf.c);
  const bool ut_zero = fabs(a.ut) < 1e-12;
  bool lost = false;       // a wait for the maxima ran out (control warp)
  int last = a.steps - 1;  // the sweep whose field is the result
  double delta = 0.0;      // control warp: max|du| of the last sweep tested
  // sweeps 0 .. steps-1; the trip after them only finishes the last test
  const int trips = HEAT ? a.steps : a.steps + 1;
  for (int t = 0; t < trips; ++t) {
    if (control) {
      if (t < a.steps) ex.begin(t, expect, lane);
      if (!HEAT && t >= 1) {
        const int r = (t - 1) & 3;
        const double m = warp_max_nonneg(lane < nwarps ? wmax[(t - 1) & 1][lane] : 0.0);
        if (lane == 0) mb_expect(mbc + r, 8u * csize);
        __syncwarp();
        if (lane < (int)csize)
          cl_store_async(cmax_to + 8u * (unsigned)(r * kClusterMax), m, mbc_to + 8u * (unsigned)r);
        if (!lost) lost = !mb_wait(mbc + r, (unsigned)((t - 1) >> 2) & 1u);
        delta = warp_max_nonneg(lane < (int)csize ? cmax[r][lane] : 0.0);
        int v = 0;
        if (delta < a.tol)
          v = 1 + PDEB200_OK;
        else if (iter0 + t >= a.max_iter)  // sweeps completed with sweep t - 1
          v = 1 + PDEB200_ERR_NOT_CONVERGED;
        if (lane == 0) verdict[t & 1] = v;
      }
      if (t < a.steps) ex.wait(t);
    } else if (t < a.steps) {
      const char* src = reinterpret_cast<const char*>(sm + (t & 1 ? a.buf_nodes : 0));
      char* dst = reinterpret_cast<char*>(sm + (t & 1 ? 0 : a.buf_nodes));
      const unsigned bytes = t & 1 ? 0u : 8u * (unsigned)a.buf_nodes;
      double acc = 0.0;
      // kClusterNodes nodes per trip, all computed before any is stored: a
      // node is a chain of dependent FP64 operations
      for (int q0 = tid; q0 < cnt; q0 += kClusterNodes * nt) {
        unsigned e[kClusterNodes];
        double rhs[kClusterNodes], old_u[kClusterNodes], v[kClusterNodes], center[kClusterNodes];
#pragma unroll
        for (int m = 0; m < kClusterNodes; ++m) {
          const int q = min(q0 + m * nt, cnt - 1);
          e[m] = tab[q];
          const double* c = reinterpret_cast<const double*>(src + (e[m] & kClOffMask));
          const Stencil<double> st = cf.template at<double, D>(g, (long long)s.off0 + ((e[m] & kClOffMask) >> 3));
          const double zp = D == 3 ? c[sxy] : 0.0, zm = D == 3 ? c[-sxy] : 0.0;
          old_u[m] = c[0];
          const double fv = sf[q];
          const double lap = nb_sum<double>(st, c[1], c[-1], c[nx], c[-nx], zp, zm, D);
          center[m] = st.c;
          if constexpr (HEAT) {
            const double opv = st.c * old_u[m] + lap;
            rhs[m] = -(NL ? __dadd_rn(opv + fv, nl_eval(nl, old_u[m])) : opv + fv);
          } else {
            rhs[m] = -(NL ? __dadd_rn(fv, nl_eval(nl, old_u[m])) : fv) - lap;
          }
        }
        if constexpr (HEAT || kConstCoef) {
          bool fast = div.safe;
#pragma unroll
          for (int m = 0; m < kClusterNodes; ++m) {
            fast = fast && div.in_range(rhs[m]);
            v[m] = div.fast(rhs[m]);
          }
          if (!fast)
#pragma unroll
            for (int m = 0; m < kClusterNodes; ++m) v[m] = __ddiv_rn(rhs[m], div.b);
        } else {
#pragma unroll
          for (int m = 0; m < kClusterNodes; ++m) {
            v[m] = __ddiv_rn(rhs[m], center[m]);
            if (fabs(center[m]) < 1e-12) {
              *degenerate = 1;
              v[m] = old_u[m];
            }
          }
        }
#pragma unroll
        for (int m = 0; m < kClusterNodes; ++m) {
          if constexpr (HEAT) {
            double u_t = ut_zero ? 0.0 : v[m];
            if (!isfinite(u_t)) u_t = 0.0;
            v[m] = old_u[m] + a.dt * u_t;
          }
          if (q0 + m * nt < cnt) {
            // (not of a repeated last node: another thread sends its copy, so the
            // neighbour may already be writing the next sweep's values around it)
            if constexpr (!HEAT) {
              const double du = fabs(v[m] - old_u[m]);
              if (du > acc) acc = du;
            }
            *reinterpret_cast<double*>(dst + (e[m] & kClOffMask)) = v[m];
            if (e[m] >> kClFaceShift) {
              const unsigned faces = (e[m] >> kClFaceShift) & 63u;
              if (faces) cl_close(g, face, s, reinterpret_cast<double*>(dst), (int)((e[m] & kClOffMask) >> 3), faces, v[m]);
              ex.push(t, e[m], bytes, v[m]);
            }
          }
        }
      }
      if constexpr (!HEAT) {
        acc = warp_max_nonneg(acc);
        if (lane == 0) wmax[t & 1][warp] = acc;
      }
    }
    __syncthreads();
    if (!HEAT && verdict[t & 1]) {  // set in this trip: the test of sweep t - 1
      last = t - 1;
      break;
    }
  }
  // own layers and the boundary layers next to them
  const double* res = sm + ((last + 1) & 1 ? a.buf_nodes : 0);
  for (int t = tid; t < local; t += blockDim.x) {
    const int layer = t / s.L;
    if ((layer == 0 && s.has_prev) || (layer == s.n + 1 && s.has_next)) continue;
    u[s.off0 + t] = res[t];
  }
  if (!HEAT && rank == 0 && control && lane == 0) {
    ctl->iter = iter0 + last + 1;
    ctl->delta = delta;
    const int v = verdict[(last + 1) & 1];
    if (v) {
      ctl->status = v - 1;
      ctl->stop = 1;
    }
  }
  cl_sync(csize);  // no CTA leaves while another may still write into its shared memory
  if (control && lane == 0 && (ex.dead || lost)) {
    ctl->status = PDEB200_ERR_TIMEOUT;
    ctl->done = 1;
  }
}

}  // namespace pdeb
