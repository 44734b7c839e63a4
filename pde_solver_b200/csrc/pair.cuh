// Whole red-black Gauss-Seidel sweep in one pass over memory for large 3D levels
// (k_rbgs_pair), and the apply of the same levels by columns (k_apply_columns).
//
// Two colour passes (k_rbgs) each read all of x, b and k and use half of every
// sector. One sweep needs them read once and x written once. A lane
// owns the columns (i, j0 .. j0 + R - 1) and marches through z two planes per
// step: at a node of column parity a it updates the first colour on plane
// P = p + a and the second colour on plane P - 1. Both are the lane's own
// column, so
// - the old values of the first colour are never read: one x value per step
//   and column is loaded (plane P + 1, second colour), the one below is the
//   previous step's;
// - a neighbour column has the other parity, so its old value on plane P is its
//   value below (P - 1 of the neighbour) or above, and its new first-colour
//   value on plane P - 1 is the one of this step or of the previous one: both
//   come from the neighbour's registers, by a shuffle in x, from the same lane
//   in y, through shared memory between the warps of a block (one barrier per
//   two planes);
// - every lane works in every step, whatever its colour.
// Tiles overlap by one column and row on each side, whose first colour is
// recomputed from old values: blocks never read each other's results, the sweep
// reads x_in and writes x_out, and is race free and deterministic. The update is
// that of k_rbgs. x_in's boundary entries are zero, x_out's are not written.
// ZERO: x_in is identically zero and not read. DOT: as in k_rbgs.
// Issue bound (about 110 instructions per lane and column step, 63% of the
// issue slots), then DRAM: FP32 513^3 421 us per sweep against 737 for two colour
// passes (250 at the copy rate); FP64 257^3 101 against 162, 300^3 139 against 261.
// Divergence form: k of the neighbours by shuffles too; FP64 257^3 169 us against
// 226, BF16 k in FP32 126 against 145. Lanes off the interior keep ordinary
// dividends: zeros take the division's slow branch and held whole blocks up (258
// instead of 177 in the 3 x 8 x 1 shape).
#pragma once

#include "cluster.cuh"
#include "kernels.cuh"

namespace pdeb {

constexpr int kPairCols = 30;  // columns a warp writes
// Rows per lane, warps per block and blocks per SM. FP32 at 513^3: 4 x 8 x 2
// 421 us, 4 x 4 x 5 418 (spills), 3 x 8 x 3 443, 6 x 4 x 3 425, 8 x 4 x 3 501;
// FP64 at 257^3 / 300^3: 3 x 8 x 2 101 / 139, 2 x 16 x 1 111 / 153, 2 x 8 x 2
// 107 / 152, 3 x 4 x 4 101 / 154. Divergence form at 257^3, a sweep / one from
// zero: FP64 2 x 12 x 1 169 / 135, 3 x 8 x 1 178 / 152, 2 x 8 x 2 209 (spills), 4 x 4
// x 2 183, 3 x 10 x 1 271 (spills); BF16 k 3 x 8 x 2 126 / 105, 4 x 8 x 2 131 / 113,
// 4 x 4 x 3 128 / 98, 2 x 8 x 3 130 / 105, 4 x 8 x 1 156 / 140.
template <int R_, int W_, int B_>
struct PairShapeOf {
  static constexpr int R = R_, W = W_, kMinBlocks = B_;
  static constexpr int kRows = R_ * W_ - 2;  // rows a block writes
};
template <class Coef, typename T>
using PairShape = std::conditional_t<
    std::is_same<Coef, CoefConst>::value,
    std::conditional_t<sizeof(T) == 4, PairShapeOf<4, 8, 2>, PairShapeOf<3, 8, 2>>,
    std::conditional_t<sizeof(T) == 4, PairShapeOf<3, 8, 2>, PairShapeOf<2, 12, 1>>>;

// k of divergence-form coefficients
template <class Coef>
struct PairK {
  static constexpr bool kHas = false, kOk = std::is_same<Coef, CoefConst>::value;
  static constexpr double kBytes = 0.0;
  __device__ static const float* field(const Coef&) { return nullptr; }
};
template <typename KT>
struct PairK<CoefDivk<KT>> {
  static constexpr bool kHas = true, kOk = true;
  static constexpr double kBytes = sizeof(KT);
  __device__ static const KT* field(const CoefDivk<KT>& c) { return c.k; }
};
template <typename T, typename KT>
__device__ __forceinline__ T pair_k(KT k) {
  if constexpr (std::is_same<KT, __nv_bfloat16>::value)
    return T(__bfloat162float(k));
  else
    return T(k);
}

// Closure factors c1 of the six faces (per face, 0 for Dirichlet).
struct PairFold {
  double lo[3], hi[3];
};

// Quotients by one divisor as in RoundedDiv (the general division's bits, in
// FP32 too: 2e10 random pairs each, no difference), the range test on the
// dividend's magnitude alone: an unsafe divisor makes the range empty.
template <typename T>
struct PairDiv {
  T b, y;
  __device__ __forceinline__ void init(T d, T& least) {
    b = d;
    const T m = fabs(d);
    if constexpr (sizeof(T) == 4) {
      y = __frcp_rn(d);
      if (!(m > 0x1p-40f && m < 0x1p40f) || (__float_as_uint(d) & 0x7fffffu) == 0x7fffffu) least = INFINITY;
    } else {
      RoundedDiv q;
      q.init(d);
      y = q.y;
      if (!q.safe) least = INFINITY;
    }
  }
  // for |a| in [least, kMost); 0 where y is
  __device__ __forceinline__ T operator()(T a) const {
    if constexpr (sizeof(T) == 4) {
      float q = __fmul_rn(a, y);
      q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
      return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    } else {
      double q = __dmul_rn(a, y);
      q = __fma_rn(__fma_rn(-b, q, a), y, q);
      return __fma_rn(__fma_rn(-b, q, a), y, q);
    }
  }
  static constexpr T kLeast = sizeof(T) == 4 ? T(0x1p-60) : T(0x1p-600);
  static constexpr T kMost = sizeof(T) == 4 ? T(0x1p60) : T(0x1p600);
};

template <class Coef, typename T, bool ZERO, bool DOT, class Post, class S = PairShape<Coef, T>>
__global__ void __launch_bounds__(32 * S::W, S::kMinBlocks)
    k_rbgs_pair(LevelGeo g, PairFold fold, Coef cf, const T* __restrict__ b, const T* __restrict__ xin,
                T* __restrict__ xout, int first, const Ctl* ctl, RedSlot slot, Post post) {
  if (ctl_skip_dep(ctl)) return;
  constexpr int R = S::R, W = S::W;
  constexpr bool kK = PairK<Coef>::kHas;
  constexpr int RK = kK ? R : 1;
  const auto* const kf = PairK<Coef>::field(cf);
  using KT = std::remove_cv_t<std::remove_pointer_t<decltype(kf)>>;
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ T ex[2][W][2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * kPairCols + lane, j0 = blockIdx.y * (W * R - 2) + warp * R;
  const int len = g.nz - 2, chunk = (len + gridDim.z - 1) / gridDim.z;
  const int k0 = 1 + blockIdx.z * chunk, k1 = min(g.nz - 1, k0 + chunk);
  double acc[1] = {0.0};
  if (k0 < k1) {
    const int nx = g.nx, ny = g.ny, nz = g.nz, sxy = (int)g.sxy;
    const int a0 = (i + j0 + k0 - 1 + first) & 1;  // parity of the even rows
    unsigned inm = 0, outm = 0;
    // the node of row r on its plane P, in bytes of T from (0, 0) of plane p; clamped to the grid in x and y
    unsigned ro[R];
    const int ic = min(i, nx - 1);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = j0 + r, row = warp * R + r;
      if (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2) {
        inm |= 1u << r;
        if (lane >= 1 && lane <= kPairCols && row >= 1 && row <= W * R - 2) outm |= 1u << r;
      }
      ro[r] = (unsigned)(min(j, ny - 1) * nx + ic + (((r & 1) ? !a0 : a0) ? sxy : 0)) * (unsigned)sizeof(T);
    }
    const unsigned lo = (unsigned)(min(max(j0 - 1, 0), ny - 1) * nx + ic + (a0 ? sxy : 0)) * (unsigned)sizeof(T);
    const unsigned hi =
        (unsigned)(min(j0 + R, ny - 1) * nx + ic + ((((R - 1) & 1) ? !a0 : a0) ? sxy : 0)) * (unsigned)sizeof(T);
    const bool edge = lane == 0 || lane == 31;  // one x neighbour outside the warp
    const int eo = (lane == 0 ? (ic > 0 ? -1 : 0) : (ic < nx - 1 ? 1 : 0)) * (int)sizeof(T);
    const T fxl = i == 1 ? T(fold.lo[0]) : T(0), fxh = i == nx - 2 ? T(fold.hi[0]) : T(0);
    const T fyl = T(fold.lo[1]), fyh = T(fold.hi[1]), fzl = T(fold.lo[2]), fzh = T(fold.hi[2]);
    int p = k0 - 1;

    T zm[R], vp[R];  // old value on plane P - 1, first colour on plane P - 2
    struct In {      // what a step reads: x on plane P + 1, b on P and P - 1, neighbours outside the warp on P
      T zp[R], b1[R], b2[R], xe[R], ylo, yhi;
      T kc[RK], kp[RK], ke[RK], kl[2], kh[2];  // k on P and P + 1; outside the warp on P (in y also on P - 1)
    };
    T km[RK], kb[RK];  // k on planes P - 2, P - 1
    // loads of the step at q; CL: planes clamped to the grid
    auto load = [&](In& in, int q, auto clamp) {
      constexpr bool CL = decltype(clamp)::value;
      // plane P + d of a row of parity a: its base is the same in all lanes (the
      // parity is in ro) unless it is clamped
      auto get = [&](const T* x, int a, int d, unsigned o) -> T {
        const long long plane = CL ? min(max(q + a + d, 0), nz - 1) - a : q + d;
        if constexpr (CL) return x[plane * sxy + (long long)(o / (unsigned)sizeof(T))];
        return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(x + plane * sxy) + o);
      };
      auto getk = [&](int a, int d, unsigned o) -> T {
        const long long plane = CL ? min(max(q + a + d, 0), nz - 1) - a : q + d;
        if constexpr (CL) return pair_k<T>(kf[plane * sxy + (long long)(o / (unsigned)sizeof(T))]);
        return pair_k<T>(*reinterpret_cast<const KT*>(reinterpret_cast<const char*>(kf + plane * sxy) +
                                                      o / (unsigned)(sizeof(T) / sizeof(KT))));
      };
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int a = (r & 1) ? 1 - a0 : a0;
        if constexpr (kK) {
          in.kc[r] = getk(a, 0, ro[r]);
          in.kp[r] = getk(a, 1, ro[r]);
          in.ke[r] = edge ? getk(a, 0, ro[r] + eo) : T(0);
        }
        in.zp[r] = ZERO ? T(0) : get(xin, a, 1, ro[r]);
        in.xe[r] = !ZERO && edge ? get(xin, a, 0, ro[r] + eo) : T(0);
        in.b1[r] = get(b, a, 0, ro[r]);
        in.b2[r] = get(b, a, -1, ro[r]);
      }
      in.ylo = ZERO ? T(0) : get(xin, a0, 0, lo);
      const int ah = ((R - 1) & 1) ? 1 - a0 : a0;
      in.yhi = ZERO ? T(0) : get(xin, ah, 0, hi);
      if constexpr (kK) {
        in.kl[0] = getk(a0, 0, lo);
        in.kl[1] = getk(a0, -1, lo);
        in.kh[0] = getk(ah, 0, hi);
        in.kh[1] = getk(ah, -1, hi);
      }
    };
    Stencil<T> st;
    if constexpr (!kK) st = cf.template at<T, 3>(GridDev{}, 0);
    PairDiv<T> dv[kK ? 1 : R];  // by the centre of each row with its x and y closures
    T least[kK ? 1 : R];  // range test of the dividends: below any value on other rows (their zeros are not divided)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int a = (r & 1) ? 1 - a0 : a0;
      auto pl = [&](int d) {
        return (long long)(min(max(p + a + d, 0), nz - 1) - a) * sxy + (long long)(ro[r] / (unsigned)sizeof(T));
      };
      zm[r] = ZERO ? T(0) : xin[pl(-1)];
      vp[r] = T(0);
      if constexpr (kK) {
        km[r] = pair_k<T>(kf[pl(-2)]);
        kb[r] = pair_k<T>(kf[pl(-1)]);
      } else {
        T c = st.c;
        c += st.xm * fxl;
        c += st.xp * fxh;
        if (j0 + r == 1) c += st.ym * fyl;
        if (j0 + r == ny - 2) c += st.yp * fyh;
        least[r] = PairDiv<T>::kLeast;
        dv[r].init(c, least[r]);
        if (!(inm >> r & 1)) {
          dv[r].y = T(0);
          least[r] = T(-1);
        }
      }
    }
    // Value of the node of row r on plane P with k around it (zero: of a zero field;
    // CoefDivk::at with
    // its factors 1/2 gathered, fold_faces, the general division). Other rows
    // divide their centre by itself: a zero dividend takes the slow division.
    auto from_k = [&](int r, bool zed, int P, T kc, T kxm, T kxp, T kym, T kyp, T kzm, T kzp, T bv, T xp, T xm, T yp, T ym,
                      T zpv, T zmv, auto zero) -> T {
      if constexpr (kK) {
        const T hx = T(0.5) * T(cf.ihx2), hy = T(0.5) * T(cf.ihy2), hz = T(0.5) * T(cf.ihz2);
        const T sxm = kc + kxm, sxp = kc + kxp, sym = kc + kym, syp = kc + kyp, szm = kc + kzm, szp = kc + kzp;
        Stencil<T> t;
        t.xm = -sxm * hx - T(cf.cx);
        t.xp = -sxp * hx + T(cf.cx);
        t.ym = -sym * hy - T(cf.dyc);
        t.yp = -syp * hy + T(cf.dyc);
        t.zm = -szm * hz - T(cf.dzc);
        t.zp = -szp * hz + T(cf.dzc);
        T c = (sxm + sxp) * hx + (sym + syp) * hy;
        c += (szm + szp) * hz;
        c += T(cf.e);
        c += t.xm * fxl;
        c += t.xp * fxh;
        if (j0 + r == 1) c += t.ym * fyl;
        if (j0 + r == ny - 2) c += t.yp * fyh;
        bool in = inm >> r & 1;
        if (zed) {
          if (P == 1) c += t.zm * fzl;
          if (P == nz - 2) c += t.zp * fzh;
          in = in && P >= 1 && P <= nz - 2;
        }
        T n = bv;
        if constexpr (!decltype(zero)::value) n = bv - nb_sum<T>(t, xp, xm, yp, ym, zpv, zmv, 3);
        T d = in ? n : c;
        if constexpr (sizeof(T) == 8)
          asm("" : "+d"(d));  // (the selections would be merged into one after the division)
        else
          asm("" : "+f"(d));
        const T v = d / c;
        return in ? v : T(0);
      }
      return T(0);
    };
    // numerators to values, with one range test for all rows
    auto quotients = [&](T (&v)[R]) {
      bool ok = true;
#pragma unroll
      for (int r = 0; r < R; ++r) ok = ok && fabs(v[r]) >= least[r] && fabs(v[r]) < PairDiv<T>::kMost;
      if (ok) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = dv[r](v[r]);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = inm >> r & 1 ? v[r] / dv[r].b : T(0);
      }
    };
    // near a z face: the values of interior nodes, centres with the z closures
    auto edge_quotients = [&](T (&v)[R], int pe, int po) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int P = (r & 1) ? po : pe;
        T c = dv[r].b;
        if (P == 1) c += st.zm * fzl;
        if (P == nz - 2) c += st.zp * fzh;
        v[r] = (inm >> r & 1) && P >= 1 && P <= nz - 2 ? v[r] / c : T(0);
      }
    };
    int buf = 0;
    // One step at p. HOT: every node of it is off the z faces and inside the chunk.
    auto step = [&](const In& in, In& next, auto hot) {
      constexpr bool HOT = decltype(hot)::value;
      const int pe = p + a0, po = p + 1 - a0;  // P of the even and odd rows
      if constexpr (HOT)
        load(next, p + 2, std::false_type{});
      else if (p + 2 <= k1)
        load(next, p + 2, std::true_type{});
      // node of row r on plane P + d (d = 0, -1), if this block writes it
      auto put = [&](int d, int r, T val, T rhs) {
        const int P = ((r & 1) ? po : pe) + d;
        if ((outm >> r & 1) && (HOT || (P >= k0 && P < k1))) {
          *reinterpret_cast<T*>(reinterpret_cast<char*>(xout + (long long)(p + d) * sxy) + ro[r]) = val;
          if constexpr (DOT) acc[0] += double(rhs) * double(val);
        }
      };
      T s[R], v[R], w[R], s1[RK], s2[RK];  // (s1, s2: k on the neighbours' planes P and P - 1)
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = ((r & 1) ? !a0 : a0) ? zm[r] : in.zp[r];  // as the neighbours read it
      if constexpr (kK) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool a = (r & 1) ? !a0 : a0;
          s1[r] = a ? kb[r] : in.kp[r];
          s2[r] = a ? km[r] : in.kc[r];
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        T xl = T(0), xr = T(0), yl = T(0), yh = T(0);
        if constexpr (!ZERO) {
          xl = __shfl_up_sync(kAll, s[r], 1);
          xr = __shfl_down_sync(kAll, s[r], 1);
          if (lane == 0) xl = in.xe[r];
          if (lane == 31) xr = in.xe[r];
          yl = r > 0 ? s[r > 0 ? r - 1 : 0] : in.ylo;
          yh = r < R - 1 ? s[r < R - 1 ? r + 1 : 0] : in.yhi;
        }
        if constexpr (kK) {
          T kl = __shfl_up_sync(kAll, s1[r], 1), kr = __shfl_down_sync(kAll, s1[r], 1);
          if (lane == 0) kl = in.ke[r];
          if (lane == 31) kr = in.ke[r];
          v[r] = from_k(r, !HOT, (r & 1) ? po : pe, in.kc[r], kl, kr, r > 0 ? s1[r > 0 ? r - 1 : 0] : in.kl[0],
                        r < R - 1 ? s1[r < R - 1 ? r + 1 : 0] : in.kh[0], kb[r], in.kp[r], in.b1[r], xr, xl, yh, yl,
                        in.zp[r], zm[r], std::integral_constant<bool, ZERO>{});
        } else {
          v[r] = in.b1[r];
          if constexpr (!ZERO) v[r] = in.b1[r] - nb_sum<T>(st, xr, xl, yh, yl, in.zp[r], zm[r], 3);
        }
      }
      if constexpr (kK) {
      } else if constexpr (HOT)
        quotients(v);
      else
        edge_quotients(v, pe, po);
#pragma unroll
      for (int r = 0; r < R; ++r) put(0, r, v[r], in.b1[r]);
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = ((r & 1) ? !a0 : a0) ? vp[r] : v[r];
      ex[buf][warp][0][lane] = s[0];
      ex[buf][warp][1][lane] = s[R - 1];
      __syncthreads();
      const T nlo = ex[buf][warp > 0 ? warp - 1 : 0][1][lane];
      const T nhi = ex[buf][warp < W - 1 ? warp + 1 : 0][0][lane];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const T xl = __shfl_up_sync(kAll, s[r], 1), xr = __shfl_down_sync(kAll, s[r], 1);
        const T yl = r > 0 ? s[r > 0 ? r - 1 : 0] : nlo, yh = r < R - 1 ? s[r < R - 1 ? r + 1 : 0] : nhi;
        if constexpr (kK) {
          const T kl = __shfl_up_sync(kAll, s2[r], 1), kr = __shfl_down_sync(kAll, s2[r], 1);
          w[r] = from_k(r, !HOT, ((r & 1) ? po : pe) - 1, kb[r], kl, kr, r > 0 ? s2[r > 0 ? r - 1 : 0] : in.kl[1],
                        r < R - 1 ? s2[r < R - 1 ? r + 1 : 0] : in.kh[1], km[r], in.kc[r], in.b2[r], xr, xl, yh, yl, v[r],
                        vp[r], std::false_type{});
        } else {
          w[r] = in.b2[r] - nb_sum<T>(st, xr, xl, yh, yl, v[r], vp[r], 3);
        }
      }
      if constexpr (kK) {
      } else if constexpr (HOT)
        quotients(w);
      else
        edge_quotients(w, pe - 1, po - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        put(-1, r, w[r], in.b2[r]);
        zm[r] = in.zp[r];
        vp[r] = v[r];
        if constexpr (kK) {
          km[r] = in.kc[r];
          kb[r] = in.kp[r];
        }
      }
      buf ^= 1;
      p += 2;
    };
    In A, B;
    load(A, p, std::true_type{});
    while (p <= k1) {
      // (hot: the loads of the next step need no clamping either)
      if (p > k0 && p > 2 && p + 1 < k1 && p + 4 <= nz - 1)
        step(A, B, std::true_type{});
      else
        step(A, B, std::false_type{});
      A = B;
    }
  }
  if constexpr (DOT) grid_reduce<1, false>(acc, slot, post);
}

// y = A_fold x of the same levels (MODE 0), with the sum of w y (MODE 1) or the
// sums of y y and y w (MODE 2), or y = w - A_fold x (MODE 3). A lane marches R
// rows of a column: each x value is loaded once (plus the rows and columns
// around a warp), neighbours in x by shuffles, in y and z from registers; the
// planes two ahead are in flight. FP32 513^3: 238 us (297 by k_apply_folded,
// 165 at the copy rate), residual 305 (371, 250); with the sums 380, where the
// separate dot products take another 130 to 165. FP64 300^3: 95 (111), residual no
// faster (121, 120), so that keeps k_residual_folded.
// Warps per block, rows per lane: the 513^3 mixed solve 61.0 ms with 4 x 4, 62.5 with
// 2 warps, 61.3 with 8, 63.2 with 2 rows, 62.4 with 6.
constexpr int kColW = 4, kColRows = 4;
// planes per block: without a sum short chunks spread the work, with one fewer
// blocks leave fewer partial sums (513^3 FP32 21 / 43 / 86 planes: apply 238 / 242 /
// 263 us, with a sum 415 / 378 / 387)
constexpr int kColPlanes = 21, kColPlanesSum = 48;
inline PairFold pair_fold(const GridDev& g) {
  ExtCoef e;
  ext_coef(g, &e);
  PairFold f;
  for (int a = 0; a < 3; ++a) {
    f.lo[a] = e.lo[a];
    f.hi[a] = e.hi[a];
  }
  return f;
}
template <typename T, int MODE, class Post, int R = kColRows>
__global__ void __launch_bounds__(32 * kColW) k_apply_columns(LevelGeo g, PairFold fold, CoefConst cf,
                                                              const T* __restrict__ x, const T* __restrict__ w,
                                                              T* __restrict__ y, const Ctl* ctl, RedSlot slot,
                                                              Post post) {
  if (ctl_skip_dep(ctl)) return;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NV = MODE == 1 ? 1 : (MODE == 2 ? 2 : 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = 1 + blockIdx.x * 32 + lane, j0 = 1 + (blockIdx.y * kColW + warp) * R;
  const int len = g.nz - 2, chunk = (len + gridDim.z - 1) / gridDim.z;
  const int k0 = 1 + blockIdx.z * chunk, k1 = min(g.nz - 1, k0 + chunk);
  double acc[NV > 0 ? NV : 1] = {};
  if (k0 < k1 && j0 <= g.ny - 2) {
    const int nx = g.nx, ny = g.ny, nz = g.nz, sxy = (int)g.sxy;
    const int ic = min(i, nx - 1);
    const bool edge = lane == 0 || lane == 31;
    const int eo = (lane == 0 ? -1 : (ic < nx - 1 ? 1 : 0)) * (int)sizeof(T);
    const Stencil<T> st = cf.template at<T, 3>(GridDev{}, 0);
    unsigned outm = 0, ro[R];  // bytes from (0, 0) of a plane, clamped to the grid
    T cr[R];                   // centres with the x and y closures
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = j0 + r;
      if (i <= nx - 2 && j <= ny - 2) outm |= 1u << r;
      ro[r] = (unsigned)(min(j, ny - 1) * nx + ic) * (unsigned)sizeof(T);
      T c = st.c;
      c += st.xm * (i == 1 ? T(fold.lo[0]) : T(0));
      c += st.xp * (i == nx - 2 ? T(fold.hi[0]) : T(0));
      if (j == 1) c += st.ym * T(fold.lo[1]);
      if (j == ny - 2) c += st.yp * T(fold.hi[1]);
      cr[r] = c;
    }
    const unsigned lo = (unsigned)((j0 - 1) * nx + ic) * (unsigned)sizeof(T);
    const unsigned hi = (unsigned)(min(j0 + R, ny - 1) * nx + ic) * (unsigned)sizeof(T);
    auto get = [&](const T* a, int plane, unsigned o) -> T {
      return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(a + (long long)plane * sxy) + o);
    };
    T zm[R], zc[R], zp[R], zn[R];            // planes k - 1 .. k + 2
    T xe[R], wv[R], ylo, yhi;                // of plane k, loaded one step before
#pragma unroll
    for (int r = 0; r < R; ++r) {
      zm[r] = get(x, k0 - 1, ro[r]);
      zc[r] = get(x, k0, ro[r]);
      zp[r] = get(x, k0 + 1, ro[r]);
      xe[r] = edge ? get(x, k0, ro[r] + eo) : T(0);
      wv[r] = MODE ? get(w, k0, ro[r]) : T(0);
    }
    ylo = get(x, k0, lo);
    yhi = get(x, k0, hi);
    for (int k = k0; k < k1; ++k) {
      T xen[R], wn[R], ylon, yhin;
      const int k2 = min(k + 2, nz - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        zn[r] = get(x, k2, ro[r]);
        xen[r] = edge ? get(x, k + 1, ro[r] + eo) : T(0);
        wn[r] = MODE ? get(w, k + 1, ro[r]) : T(0);
      }
      ylon = get(x, k + 1, lo);
      yhin = get(x, k + 1, hi);
      const bool zed = k == 1 || k == nz - 2;
      T* const yk = y + (long long)k * sxy;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        T xl = __shfl_up_sync(kAll, zc[r], 1), xr = __shfl_down_sync(kAll, zc[r], 1);
        if (lane == 0) xl = xe[r];
        if (lane == 31) xr = xe[r];
        T c = cr[r];
        if (zed) {
          if (k == 1) c += st.zm * T(fold.lo[2]);
          if (k == nz - 2) c += st.zp * T(fold.hi[2]);
        }
        const T yl = r > 0 ? zc[r > 0 ? r - 1 : 0] : ylo, yh = r < R - 1 ? zc[r < R - 1 ? r + 1 : 0] : yhi;
        T v = c * zc[r] + nb_sum<T>(st, xr, xl, yh, yl, zp[r], zm[r], 3);
        if (MODE == 3) v = wv[r] - v;
        if (outm >> r & 1) {
          *reinterpret_cast<T*>(reinterpret_cast<char*>(yk) + ro[r]) = v;
          if constexpr (MODE == 1) acc[0] += double(wv[r]) * double(v);
          if constexpr (MODE == 2) {
            acc[0] += double(v) * double(v);
            acc[NV - 1] += double(v) * double(wv[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        zm[r] = zc[r];
        zc[r] = zp[r];
        zp[r] = zn[r];
        xe[r] = xen[r];
        wv[r] = wn[r];
      }
      ylo = ylon;
      yhi = yhin;
    }
  }
  if constexpr (NV > 0) grid_reduce<NV, false>(acc, slot, post);
}

}  // namespace pdeb
