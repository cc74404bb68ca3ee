// MPDATA step in a few launches under any boundary condition.
//
// The reference-structured path (general.cu) runs one kernel per formula and per
// halo fill: about 47 launches for a 2D step with FCT and open boundaries, 70 in
// 3D, each reading and writing whole arrays.  Here a step of n_iters passes is
//   k_upwind    psi1 = donor-cell(psi, GC)                    (mpdata_osc_{1,2,3}d.hpp)
// and for every corrective pass
//   k_antidiff  all components of the antidiffusive velocity  (formulae_mpdata_{1,2,3}d.hpp)
//   k_betas     FCT limiters of every cell, psi_min / psi_max in place
//               (formulae_mpdata_fct_{1,2,3}d.hpp, mpdata_fct_{1,2,3}d.hpp)
//   k_correct   limited velocities, their fluxes and the donor-cell sum
// with the arithmetic of general.cu's functors, in their order (compiled without
// FMA contraction: the same bits).  No kernel fills halos: a point outside the
// domain is read where its fill would have copied it from (scalars: cyclic wrap,
// open edge value, rigid mirror; antidiffusive velocities: the fills of
// solver_{1,2,3}d.hpp xchng_vctr_alng(.., ad) and xchng_vctr_nrml(.., 0)).  Only the
// advector keeps its halo in memory, filled once by general<T>::ante_loop.
//
// What bounds it: small grids, the launches, which overlap the previous kernel's end
// (launch_dependent: 101 x 101 open cone 21.7 -> 13.6 us per step); large grids, the
// traffic between the stages, 26 fields per step with FCT, in cache below about
// 100 MB.  The last axis lies along the warp, threads walk along the first; faces and
// limiter cells at and outside the domain's faces are further blocks of the same
// launch, so that the interior stays aligned and free of their rules.
#pragma once

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "stages.cuh"

namespace mpdx {
namespace sg {

template <class T> struct lim;
template <> struct lim<float> {
  __device__ static float tiny() { return FLT_MIN; }
  __device__ static float eps() { return FLT_EPSILON; }
};
template <> struct lim<double> {
  __device__ static double tiny() { return DBL_MIN; }
  __device__ static double eps() { return DBL_EPSILON; }
};
template <class T> __device__ __forceinline__ T pos(T x) { return T(0) < x ? x : T(0); }  // std::max(0, x)
template <class T> __device__ __forceinline__ T neg(T x) { return x < T(0) ? x : T(0); }  // std::min(0, x)
template <class T> __device__ __forceinline__ T dmax(T a, T b) { return a < b ? b : a; }  // std::max
template <class T> __device__ __forceinline__ T dmin(T a, T b) { return b < a ? b : a; }  // std::min
template <class T> __device__ __forceinline__ T flux(T c, T l, T r) { return pos(c) * l + neg(c) * r; }

// x / 3 and x / 6, correctly rounded without a division (mpdx::qdiv)
template <class T> __device__ __forceinline__ T div3(T x) { return qdiv<T>(x, T(3), T(1) / T(3)); }
template <class T> __device__ __forceinline__ T div6(T x) { return qdiv<T>(x, T(6), T(1) / T(6)); }

// a field by 32-bit element strides
template <class T>
struct arr {
  fptr<T> o;
  int s0, s1;  // strides of axes 0 and 1 (the last axis: 1)
};

template <class T>
struct eqn {
  arr<T> in, out;             // psi of the pass, its result
  arr<T> psin;                // psi of the step's start (k_betas)
  arr<T> corr[3], unco[3];    // antidiffusive velocity, advector it corrects
  arr<T> bu, bd, mn, mx;
};
template <class T>
struct args {
  eqn<T> e[kStageEqns];
  int n[3], bc[3][2];
};

template <int V> struct ic { static constexpr int value = V; };

// ---- coordinates ----
template <int ND, class T>
__device__ __forceinline__ int at(const arr<T> &f, int x, int y, int z) {
  if (ND == 1) return x;
  if (ND == 2) return x * f.s0 + y;
  return x * f.s0 + y * f.s1 + z;
}
template <int ND, class T>
__device__ __forceinline__ int at(const arr<T> &f, const int *c) { return at<ND>(f, c[0], c[1], c[2]); }

// where coordinate q of axis d, at most 2 outside, takes a scalar from
template <class T>
__device__ __forceinline__ int src(const args<T> &A, int d, int q) {
  const int n = A.n[d];
  if (q >= 0 && q < n) return q;
  const int side = q < 0 ? 0 : 1, kind = A.bc[d][side];
  if (kind == MPDX_BC_CYCLIC) return side ? q - (n - 1) : q + (n - 1);
  if (kind == MPDX_BC_OPEN) return side ? n - 1 : 0;
  return side ? 2 * (n - 1) - q : -q;  // rigid: mirror about the wall point
}
// the same for a transverse axis of a velocity component; false where its fill is zero
template <class T>
__device__ __forceinline__ bool vsrc(const args<T> &A, int d, int &q) {
  if (q >= 0 && q < A.n[d]) return true;
  if (A.bc[d][q < 0 ? 0 : 1] == MPDX_BC_OPEN) return false;
  q = src(A, d, q);
  return true;
}

// point of a 1D grid owned by this thread (false: none)
template <int ND, class T>
__device__ __forceinline__ bool own(const args<T> &A, int c[3]) {
  c[0] = blockIdx.x * blockDim.x + threadIdx.x;
  c[1] = c[2] = 0;
  return c[0] < A.n[0];
}
// index into the list that the blocks from nb on work through
__device__ __forceinline__ long long list_index(int nb) {
  return ((long long)(blockIdx.x - nb) * gridDim.y + blockIdx.y) * blockDim.x + threadIdx.x;
}
// entry q of the list of faces of the grid: axis d, position in the plane across it
// (its two axes in order); false beyond the list.  Axis after axis, n_sides entries
// per position.
template <int ND, class T>
__device__ __forceinline__ bool face_entry(const args<T> &A, long long q, int n_sides, int &d, int &side, int c[3]) {
#pragma unroll
  for (d = 0; d < ND; ++d) {
    const int a = d == 0 ? 1 : 0, b = d == 2 ? 1 : 2;  // the other axes
    const int na = ND > 1 ? A.n[a] : 1, nb = ND > 2 ? A.n[b] : 1;
    const long long m = (long long)na * nb;
    if (q < m * n_sides) {
      side = q >= m ? 1 : 0;
      const int w = int(q - (side ? m : 0));
      c[0] = c[1] = c[2] = 0;
      if (ND > 1) c[a] = w / nb;
      if (ND > 2) c[b] = w - c[a] * nb;
      return true;
    }
    q -= m * n_sides;
  }
  return false;
}

// Threads per block: 128; with 256 the waits at the ends of blocks cost 2 to 9 % more
// (1024^2 in three passes 103.5 and 95.6 us per step, 256 x 256 x 128 FP32 371 and 359).
constexpr int kStageThreads = 128;
// Blocks per SM that the registers are kept for: the kernels wait on L2 and DRAM, and
// the walk's carried values would otherwise leave 8 warps per SM (k_antidiff at 150
// registers).  250 x 257 x 241 iga|fct, us per step without and with: FP64 1240 and 996,
// FP32 657 and 633.  The limits make most of the 3D kernels spill, which costs less than
// the warps are worth.  Bytes stored and loaded per thread, FP64: k_upwind 40 / 96;
// k_antidiff 4 / 4 (iga) to 176 / 252 (tot without iga); k_betas 40 / 68 to 64 / 108;
// k_correct with the limiter 132 / 132 (iga), 268 / 408 (without); FP32: k_antidiff up to
// 84 / 88 (iga|tot), k_correct 68 / 128.
template <class T> struct blocks;
template <> struct blocks<float> { static constexpr int upwind = 10, antidiff = 6, betas = 8, correct = 10; };
template <> struct blocks<double> { static constexpr int upwind = 12, antidiff = 4, betas = 8, correct = 12; };

// The march of the 2D and 3D kernels: a thread owns a position of the axes after the
// first and walks `mi` planes along axis 0, so that positions, halo rules and offsets
// across are worked out once, those along axis 0 are the same for a whole block, and
// values of the last planes stay in registers (k_antidiff reads 19 values per point
// instead of 35 to 40).  One thread per point instead: 288, 392, 384 and 252
// instructions per point in the four kernels, 1159 us per step at 256^3 in FP64.
struct walk {
  int j, k, i0, i1;
};
template <int ND, class T>
__device__ __forceinline__ bool column(const args<T> &A, int mi, walk &w) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, pos = ND == 3 ? A.n[1] * A.n[2] : A.n[1];
  if (p >= pos) return false;
  w.j = ND == 3 ? int(unsigned(p) / unsigned(A.n[2])) : p;
  w.k = ND == 3 ? p - w.j * A.n[2] : 0;
  w.i0 = blockIdx.y * mi;
  w.i1 = min(w.i0 + mi, A.n[0]);
  return w.i0 < w.i1;
}
// offset of a position in a plane of f
template <int ND, class T>
__device__ __forceinline__ int in_plane(const arr<T> &f, int j, int k) { return ND == 3 ? j * f.s1 + k : j; }

// ---- donor cell ----
// fluxes through the two faces of a cell along axis d under the rigid rule for
// fluxes (xchng_flux): F(-1) = -F(0), F(n-1) = -F(n-2)
template <class T, class F>
__device__ __forceinline__ T net(const args<T> &A, int d, int c, F &&f) {  // -F(+1/2) + F(-1/2)
  T hi = f(0), lo = f(-1);
  if (c == 0 && A.bc[d][0] == MPDX_BC_RIGID) lo = -hi;
  else if (c == A.n[d] - 1 && A.bc[d][1] == MPDX_BC_RIGID) hi = -lo;
  return -hi + lo;
}
template <int ND, class T>
__device__ __forceinline__ T donor(T p, const T *nt) {
  if (ND == 1) return p + nt[0];
  if (ND == 2) return p + (nt[0] + nt[1]);
  return p + (nt[0] + nt[1] + nt[2]);
}

template <int ND, class T>
__global__ void __launch_bounds__(kStageThreads, blocks<T>::upwind) k_upwind(const __grid_constant__ args<T> A, int mi) {
  next_may_start();
  const eqn<T> &E = A.e[blockIdx.z];
  if constexpr (ND == 1) {
    int c[3];
    if (!own<ND>(A, c)) return;
    after_previous();
    const auto p = E.in.o, g = E.unco[0].o;
    const T p0 = p[c[0]], pp = p[src(A, 0, c[0] + 1)], pm = p[src(A, 0, c[0] - 1)], g1 = g[c[0]], g0 = g[c[0] - 1];
    const T nt = net(A, 0, c[0], [&](int f) { return f == 0 ? flux(g1, p0, pp) : flux(g0, pm, p0); });
    E.out.o[c[0]] = p0 + nt;
  } else {
    walk w;
    if (!column<ND>(A, mi, w)) return;
    const int j = w.j, k = w.k;
    const int o = in_plane<ND>(E.in, j, k), oj = in_plane<ND>(E.in, src(A, 1, j + 1), k), ojm = in_plane<ND>(E.in, src(A, 1, j - 1), k);
    const int ok = ND == 3 ? in_plane<ND>(E.in, j, src(A, 2, k + 1)) : 0, okm = ND == 3 ? in_plane<ND>(E.in, j, src(A, 2, k - 1)) : 0;
    const arr<T> &F0 = E.unco[0], &F1 = E.unco[1], &F2 = E.unco[ND - 1];
    const int a0 = in_plane<ND>(F0, j, k), a1 = in_plane<ND>(F1, j, k), a2 = in_plane<ND>(F2, j, k), s1 = ND == 3 ? F1.s1 : 1;
    auto plane = [&](const arr<T> &f, int i) { return f.o + (long long)i * f.s0; };
    after_previous();
    T p0 = plane(E.in, w.i0)[o];
    T lo = flux(plane(F0, w.i0 - 1)[a0], plane(E.in, src(A, 0, w.i0 - 1))[o], p0);
#pragma unroll 2
    for (int i = w.i0; i < w.i1; ++i) {
      const auto q = plane(E.in, i), q1 = plane(F1, i);
      const T pn = plane(E.in, src(A, 0, i + 1))[o], g0 = plane(F0, i)[a0];
      const T pj = q[oj], pjm = q[ojm], g1 = q1[a1], g1m = q1[a1 - s1];
      T nt[3];
      const T hi = flux(g0, p0, pn);
      nt[0] = net(A, 0, i, [&](int f) { return f == 0 ? hi : lo; });
      nt[1] = net(A, 1, j, [&](int f) { return f == 0 ? flux(g1, p0, pj) : flux(g1m, pjm, p0); });
      if constexpr (ND == 3) {
        const auto q2 = plane(F2, i);
        const T pk = q[ok], pkm = q[okm], g2 = q2[a2], g2m = q2[a2 - 1];
        nt[2] = net(A, 2, k, [&](int f) { return f == 0 ? flux(g2, p0, pk) : flux(g2m, pkm, p0); });
      }
      E.out.o[(long long)i * E.out.s0 + o] = donor<ND>(p0, nt);
      lo = hi;
      p0 = pn;
    }
  }
}

// ---- antidiffusive velocity ----
template <class T> __device__ __forceinline__ T frac(T nom, T den) { return nom / (den + lim<T>::tiny()); }
template <bool IGA, class T> __device__ __forceinline__ T nd4(T a, T b, T c, T d) {
  if (IGA) return (a + b - c - d) / T(4);
  return frac(a + b - c - d, a + b + c + d);
}
template <bool IGA, class T> __device__ __forceinline__ T nd2(T a, T b, T c, T d) {
  if (IGA) return T(2) * (a - b - c + d) / T(4);
  return T(2) * frac(a - b - c + d, a + b + c + d);
}
template <class T> __device__ __forceinline__ T cxx(T C) { return div6(T(3) * C * fabs(C) - T(2) * (C * C * C) - C); }
template <class T> __device__ __forceinline__ T cxy(T C, T g) { return (fabs(C) - T(2) * (C * C)) * g / T(2); }

// Antidiffusive velocity through one face: C its Courant number, gc1 / gc2 the averages
// of the other components around it, ps(a, b, e) psi at offsets along the face's axis
// and the two axes after it (cyclically).
template <int ND, bool IGA, bool TOT, class T, class F>
__device__ __forceinline__ T antidiff_core(T C, T gc1, T gc2, F &&ps) {
  const T p1 = ps(1, 0, 0), p0 = ps(0, 0, 0);
  T ndx;
  if (IGA) ndx = ND == 3 ? p1 - p0 : T(2) * (p1 - p0) / T(2);
  else ndx = T(2) * frac(p1 - p0, p1 + p0);
  T r = fabs(C) / T(2) * (T(1) - fabs(C)) * ndx;
  T xx = T(0);
  if (TOT) xx = nd2<IGA>(ps(2, 0, 0), p1, p0, ps(-1, 0, 0));
  if constexpr (ND == 1) {
    if (TOT) r = r + xx * cxx(C);
  } else if constexpr (ND == 2) {
    const T a = ps(1, 1, 0), b = ps(0, 1, 0), e = ps(1, -1, 0), f = ps(0, -1, 0);
    r = r - C * gc1 / T(2) * nd4<IGA>(a, b, e, f);
    if (TOT) r = r + (xx * cxx(C) + nd2<IGA>(a, b, e, f) * cxy(C, gc1));
  } else {
    const T a = ps(1, 1, 0), b = ps(0, 1, 0), e = ps(1, -1, 0), f = ps(0, -1, 0);
    const T a2 = ps(1, 0, 1), b2 = ps(0, 0, 1), e2 = ps(1, 0, -1), f2 = ps(0, 0, -1);
    r = r - C / T(2) * (gc1 * nd4<IGA>(a, b, e, f) + gc2 * nd4<IGA>(a2, b2, e2, f2));
    if (TOT) {
      const T q0 = ps(1, 1, 1), q1 = ps(1, -1, -1), q2 = ps(1, 1, -1), q3 = ps(1, -1, 1);
      const T q4 = ps(0, 1, 1), q5 = ps(0, -1, -1), q6 = ps(0, 1, -1), q7 = ps(0, -1, 1);
      const T nom = q0 + q1 - q2 - q3 + q4 + q5 - q6 - q7;
      const T yz = IGA ? nom / T(8) : frac(nom, q0 + q1 + q2 + q3 + q4 + q5 + q6 + q7);
      r = r + (xx * cxx(C) + nd2<IGA>(a, b, e, f) * cxy(C, gc1) + nd2<IGA>(a2, b2, e2, f2) * cxy(C, gc2)
               + yz * div3(T(-2) * C * gc1 * gc2));
    }
  }
  return r;
}

// component D at the face c[D] + 1/2, from psi at x[d][m + 1] for coordinate c[d] + m
// (m = -1 .. 2 along D, -1 .. 1 across), its own advector component at c, and the
// transverse components at coordinate v[m] along D for m = 0, 1 (z[m]: they are zero)
template <int ND, int D, bool IGA, bool TOT, class T>
__device__ __forceinline__ T antidiff(const eqn<T> &E, const int c[3], const int (&x)[3][4], const int (&v)[2], const bool (&z)[2]) {
  constexpr int D1 = (D + 1) % ND, D2 = (D + 2) % ND;
  auto ps = [&](int a, int b, int e) {
    int w[3] = {0, 0, 0};
    w[D] = x[D][a + 1];
    if (ND > 1) w[D1] = x[D1][b + 1];
    if (ND > 2) w[D2] = x[D2][e + 1];
    return E.in.o[at<ND>(E.in, w)];
  };
  auto bar = [&](auto qq) {  // average of component q over the four faces around
    constexpr int q = decltype(qq)::value;
    auto gq = [&](int a, int b) {
      if (z[a]) return T(0);
      int w[3] = {c[0], c[1], c[2]};
      w[D] = v[a];
      w[q] = c[q] + b;
      return E.unco[q].o[at<ND>(E.unco[q], w)];
    };
    return (gq(1, 0) + gq(0, 0) + gq(1, -1) + gq(0, -1)) / T(4);
  };
  T gc1 = T(0), gc2 = T(0);
  if constexpr (ND > 1) gc1 = bar(ic<D1>{});
  if constexpr (ND > 2) gc2 = bar(ic<D2>{});
  return antidiff_core<ND, IGA, TOT>(E.unco[D].o[at<ND>(E.unco[D], c)], gc1, gc2, ps);
}

// Component D at c (c[D] = -1 .. n-1), stored.  HALO: the advector being corrected has
// its halo in memory (the solver's own); otherwise it is the velocity of the previous
// pass, read by the rule of its fill.  With fct the faces -1 and n-1 get what the
// along-axis fill leaves there: a cyclic axis the copies of faces n-2 and 0 (evaluated
// there), an open neighbouring side zero on the edges of the domain.
template <int ND, int D, bool IGA, bool TOT, bool HALO, class T>
__device__ __forceinline__ void antidiff_face(const args<T> &A, const eqn<T> &E, const int c[3], bool fct) {
  int cc[3] = {c[0], c[1], c[2]}, x[3][4], v[2];
  bool zero = false, z[2] = {false, false};
  if (fct) {
    const int n = A.n[D];
    if (A.bc[D][0] == MPDX_BC_CYCLIC) {
      if (c[D] == -1) cc[D] = n - 2;
      else if (c[D] == n - 1) cc[D] = 0;
    } else if (c[D] == -1 || c[D] == n - 1) {
#pragma unroll
      for (int d = 0; d < D; ++d)
        zero = zero || (c[d] == 0 && A.bc[d][0] == MPDX_BC_OPEN) || (c[d] == A.n[d] - 1 && A.bc[d][1] == MPDX_BC_OPEN);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int m = -1; m <= 2; ++m) x[d][m + 1] = d >= ND || (m == 2 && !(TOT && d == D)) ? 0 : src(A, d, cc[d] + m);
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    v[m] = cc[D] + m;
    if (!HALO) z[m] = !vsrc(A, D, v[m]);
  }
  const T r = antidiff<ND, D, IGA, TOT>(E, cc, x, v, z);
  E.corr[D].o[at<ND>(E.corr[D], c)] = zero ? T(0) : r;
}

template <int ND, bool IGA, bool TOT, bool HALO, class T>
__global__ void __launch_bounds__(kStageThreads, blocks<T>::antidiff) k_antidiff(const __grid_constant__ args<T> A, int nb, int mi, bool fct) {
  next_may_start();
  const eqn<T> &E = A.e[blockIdx.z];
  if (ND == 1 || int(blockIdx.x) >= nb) {
    int c[3];
    after_previous();
    if (ND == 1 && int(blockIdx.x) < nb) {
      if (own<ND>(A, c)) antidiff_face<ND, 0, IGA, TOT, HALO>(A, E, c, fct);
      return;
    }
    int d, side;
    if (!face_entry<ND>(A, list_index(nb), fct && ND > 1 ? 2 : 1, d, side, c)) return;
    c[d] = side ? A.n[d] - 1 : -1;
    if (d == 0) antidiff_face<ND, 0, IGA, TOT, HALO>(A, E, c, fct);
    if constexpr (ND > 1) if (d == 1) antidiff_face<ND, 1, IGA, TOT, HALO>(A, E, c, fct);
    if constexpr (ND > 2) if (d == 2) antidiff_face<ND, 2, IGA, TOT, HALO>(A, E, c, fct);
    return;
  }
  if constexpr (ND > 1) {
    walk w;
    if (!column<ND>(A, mi, w)) return;
    const int j = w.j, k = w.k;
    // psi: offsets of the 3 x 3 positions around, of two beyond
    int o[3][3], o2j = 0, o2k = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        o[a][b] = ND == 3 ? in_plane<ND>(E.in, src(A, 1, j + a - 1), src(A, 2, k + b - 1)) : src(A, 1, j + a - 1);
    if (TOT) o2j = in_plane<ND>(E.in, src(A, 1, j + 2), k);
    if (TOT && ND == 3) o2k = in_plane<ND>(E.in, j, src(A, 2, k + 2));
    // velocity components one position further across (zero: nothing there)
    int jv = j + 1, kv = k + 1;
    bool zj = false, zk = false;
    if (!HALO) {
      zj = !vsrc(A, 1, jv);
      if (ND == 3) zk = !vsrc(A, 2, kv);
    }
    const arr<T> &F0 = E.unco[0], &F1 = E.unco[1], &F2 = E.unco[ND - 1];
    const int s1 = ND == 3 ? F1.s1 : 1;
    const int a0 = in_plane<ND>(F0, j, k), a0j = in_plane<ND>(F0, jv, k), a0k = ND == 3 ? in_plane<ND>(F0, j, kv) : 0;
    const int a1 = in_plane<ND>(F1, j, k), a1k = ND == 3 ? in_plane<ND>(F1, j, kv) : 0;
    const int a2 = ND == 3 ? in_plane<ND>(F2, j, k) : 0, a2j = ND == 3 ? in_plane<ND>(F2, jv, k) : 0;
    const bool last_j = fct && j == A.n[1] - 1, last_k = fct && ND == 3 && k == A.n[ND - 1] - 1;
    auto plane = [&](const arr<T> &f, int i) { return f.o + (long long)i * f.s0; };
    T P[3][3][3], g0c, g0j, g0k = T(0), h1 = T(0), h1m = T(0), h2 = T(0), h2m = T(0);
    auto load = [&](T (&Q)[3][3], int i) {
      const auto q = plane(E.in, src(A, 0, i));
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
          if (ND == 3 || b == 1) Q[a][b] = q[o[a][b]];
    };
    after_previous();
    load(P[0], w.i0 - 1);
    load(P[1], w.i0);
    {
      const auto q = plane(F0, w.i0 - 1);
      g0c = q[a0];
      g0j = zj ? T(0) : q[a0j];
      if (ND == 3) g0k = zk ? T(0) : q[a0k];
      const auto r = plane(F1, w.i0);
      h1 = r[a1]; h1m = r[a1 - s1];
      if (ND == 3) { const auto t = plane(F2, w.i0); h2 = t[a2]; h2m = t[a2 - 1]; }
    }
#pragma unroll 2
    for (int i = w.i0; i < w.i1; ++i) {
      load(P[2], i + 1);
      // along axis 0: the other components one plane further
      int iv = i + 1;
      bool zi = false;
      if (!HALO) zi = !vsrc(A, 0, iv);
      const auto q0 = plane(F0, i), q1 = plane(F1, i), n1 = plane(F1, iv), q2 = plane(F2, i), n2 = plane(F2, iv);
      const T c0 = q0[a0], c0j = zj ? T(0) : q0[a0j];
      T c0k = T(0), c1k = T(0), c1km = T(0), c2j = T(0), c2jm = T(0), m2 = T(0), m2m = T(0);
      const T m1 = zi ? T(0) : n1[a1], m1m = zi ? T(0) : n1[a1 - s1];
      if (ND == 3) {
        c0k = zk ? T(0) : q0[a0k];
        c1k = zk ? T(0) : q1[a1k];
        c1km = zk ? T(0) : q1[a1k - s1];
        c2j = zj ? T(0) : q2[a2j];
        c2jm = zj ? T(0) : q2[a2j - 1];
        m2 = zi ? T(0) : n2[a2];
        m2m = zi ? T(0) : n2[a2 - 1];
      }
      T pi2 = T(0), pj2 = T(0), pk2 = T(0);
      if (TOT) {
        pi2 = plane(E.in, src(A, 0, i + 2))[o[1][1]];
        pj2 = plane(E.in, i)[o2j];
        if (ND == 3) pk2 = plane(E.in, i)[o2k];
      }
      const T b1x = (m1 + h1 + m1m + h1m) / T(4), b2x = (m2 + h2 + m2m + h2m) / T(4);
      const T rx = antidiff_core<ND, IGA, TOT>(c0, b1x, b2x, [&](int a, int b, int e) { return a == 2 ? pi2 : P[a + 1][b + 1][e + 1]; });
      T ry;
      if (ND == 2) {
        const T b = (c0j + c0 + g0j + g0c) / T(4);
        ry = antidiff_core<ND, IGA, TOT>(h1, b, T(0), [&](int a, int b_, int) { return a == 2 ? pj2 : P[b_ + 1][a + 1][1]; });
      } else {
        const T b1 = (c2j + h2 + c2jm + h2m) / T(4), b2 = (c0j + c0 + g0j + g0c) / T(4);
        ry = antidiff_core<ND, IGA, TOT>(h1, b1, b2, [&](int a, int b, int e) { return a == 2 ? pj2 : P[e + 1][a + 1][b + 1]; });
      }
      const int ix = at<ND>(E.corr[0], i, j, k), iy = at<ND>(E.corr[1], i, j, k);
      if (!(fct && i == A.n[0] - 1)) E.corr[0].o[ix] = rx;
      if (!last_j) E.corr[1].o[iy] = ry;
      if constexpr (ND == 3) {
        const T b1 = (c0k + c0 + g0k + g0c) / T(4), b2 = (c1k + h1 + c1km + h1m) / T(4);
        const T rz = antidiff_core<ND, IGA, TOT>(h2, b1, b2, [&](int a, int b, int e) { return a == 2 ? pk2 : P[b + 1][e + 1][a + 1]; });
        if (!last_k) E.corr[2].o[at<ND>(E.corr[2], i, j, k)] = rz;
      }
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) { P[0][a][b] = P[1][a][b]; P[1][a][b] = P[2][a][b]; }
      g0c = c0; g0j = c0j; g0k = c0k;
      h1 = m1; h1m = m1m; h2 = m2; h2m = m2m;
    }
  }
}

// ---- FCT limiters ----
// antidiffusive velocity d one face beyond the stored ones (c[d] = -2 or n), the other
// coordinates interior: the along-axis fill with ad (bcond/{cyclic,open,rigid}_*.hpp)
template <int ND, int D, class T>
__device__ __forceinline__ T beyond(const args<T> &A, const eqn<T> &E, int side, const int c[3]) {
  const int n = A.n[D], kind = A.bc[D][side];
  int w[3] = {c[0], c[1], c[2]};
  const arr<T> &f = E.corr[D];
  if (kind == MPDX_BC_CYCLIC) { w[D] = side ? 1 : n - 3; return f.o[at<ND>(f, w)]; }
  if (kind == MPDX_BC_RIGID) { w[D] = side ? n - 2 : 1; return -f.o[at<ND>(f, w)]; }
  if (ND == 1) { w[D] = side ? n - 3 : 0; return f.o[at<ND>(f, w)]; }  // open_1d.hpp with a halo of 2
  const int e = side ? n - 1 : 0;
  w[D] = side ? e - 1 : e;
  T r = f.o[at<ND>(f, w)];
  w[D] = e;
  // zero divergence in the edge cell; the components after D are zero on the edges of
  // the domain at this point of the fill's order
  auto across = [&](auto qq) {
    constexpr int q = decltype(qq)::value;
    const arr<T> &g = E.corr[q];
    int lo[3] = {w[0], w[1], w[2]};
    lo[q] = w[q] - 1;
    const T a = q > D && lo[q] == -1 ? T(0) : g.o[at<ND>(g, lo)];
    const T b = q > D && w[q] == A.n[q] - 1 ? T(0) : g.o[at<ND>(g, w)];
    return a - b;
  };
  if constexpr (ND > 1) r = side ? r + across(ic<(D + 1) % ND>{}) : r - across(ic<(D + 1) % ND>{});
  if constexpr (ND > 2) r = side ? r + across(ic<(D + 2) % ND>{}) : r - across(ic<(D + 2) % ND>{});
  return r;
}

// psi_min / psi_max of a cell from psi of the step's start at the cell and its neighbours
template <int ND, class T>
__device__ __forceinline__ void bounds(T q0, const T *l, const T *h, T &mn, T &mx) {
  if (ND == 1) {
    mn = dmin(dmin(l[0], q0), h[0]);
    mx = dmax(dmax(l[0], q0), h[0]);
  } else if (ND == 2) {
    mn = dmin(dmin(dmin(dmin(h[1], l[0]), q0), h[0]), l[1]);
    mx = dmax(dmax(dmax(dmax(h[1], l[0]), q0), h[0]), l[1]);
  } else {
    mn = dmin(dmin(dmin(dmin(dmin(dmin(q0, h[0]), l[0]), h[1]), l[1]), h[2]), l[2]);
    mx = dmax(dmax(dmax(dmax(dmax(dmax(q0, h[0]), l[0]), h[1]), l[1]), h[2]), l[2]);
  }
}
// beta_up / beta_dn of a cell: psi1 at it and its neighbours, bounds, velocities (or
// fluxes) through its faces
template <int ND, class T>
__device__ __forceinline__ void betas(T p0, const T *pl, const T *ph, T mn, T mx, const T *lo, const T *hi, T &bu, T &bd) {
  T du, dd;
  if (ND == 1) {
    mx = dmax(mx, dmax(pl[0], dmax(p0, ph[0])));
    mn = dmin(mn, dmin(pl[0], dmin(p0, ph[0])));
    du = pos(lo[0]) - neg(hi[0]);
    dd = pos(hi[0]) - neg(lo[0]);
  } else if (ND == 2) {
    mx = dmax(mx, dmax(ph[1], dmax(pl[0], dmax(p0, dmax(ph[0], pl[1])))));
    mn = dmin(mn, dmin(ph[1], dmin(pl[0], dmin(p0, dmin(ph[0], pl[1])))));
    du = (pos(lo[0]) - neg(hi[0])) + (pos(lo[1]) - neg(hi[1]));
    dd = (pos(hi[0]) - neg(lo[0])) + (pos(hi[1]) - neg(lo[1]));
  } else {
    mx = dmax(mx, dmax(p0, dmax(ph[0], dmax(pl[0], dmax(ph[1], dmax(pl[1], dmax(ph[2], pl[2])))))));
    mn = dmin(mn, dmin(ph[1], dmin(pl[0], dmin(p0, dmin(ph[0], dmin(ph[2], dmin(pl[2], pl[1])))))));
    du = (pos(lo[0]) - neg(hi[0])) + (pos(lo[1]) - neg(hi[1])) + (pos(lo[2]) - neg(hi[2]));
    dd = (pos(hi[0]) - neg(lo[0])) + (pos(hi[1]) - neg(lo[1])) + (pos(hi[2]) - neg(lo[2]));
  }
  bu = (mx - p0) / (du + lim<T>::eps());
  bd = (p0 - mn) / (dd + lim<T>::eps());
}

// MODE 0: psi_min / psi_max from psin; 1: the same, and stored for the next pass; 2: as
// stored.  c: a cell of the interior, or one just outside along axis `out` (-1: none).
template <int ND, bool IGA, int MODE, class T>
__device__ __forceinline__ void beta_cell(const args<T> &A, const eqn<T> &E, const int c[3], int out) {
  int x[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int m = 0; m < 3; ++m) x[d][m] = d >= ND ? 0 : src(A, d, c[d] + m - 1);
  auto off = [&](int d, int m) {  // one step along d
    int w[3] = {x[0][1], x[1][1], x[2][1]};
    if (d < ND) w[d] = x[d][m + 1];
    return at<ND>(E.in, w);
  };
  const int o0 = off(3, 0);
  int oh[3], ol[3];
  T ph[3], pl[3];
  const T p0 = E.in.o[o0];
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    oh[d] = off(d, 1); ol[d] = off(d, -1);
    ph[d] = E.in.o[oh[d]]; pl[d] = E.in.o[ol[d]];
  }
  // velocities through the upper and lower face along each axis
  T hi[3], lo[3];
  auto faces = [&](auto dd) {
    constexpr int d = decltype(dd)::value;
    const arr<T> &f = E.corr[d];
    int w[3] = {c[0], c[1], c[2]};
    bool zero = false;
    if (out >= 0 && out != d) zero = !vsrc(A, out, w[out]);
    const int ow = at<ND>(f, w), sd = d == ND - 1 ? 1 : (d == 0 ? f.s0 : f.s1);
    if (out == d) {
      const int side = c[d] < 0 ? 0 : 1;
      hi[d] = side ? beyond<ND, d>(A, E, 1, c) : f.o[ow];
      lo[d] = side ? f.o[ow - sd] : beyond<ND, d>(A, E, 0, c);
    } else {
      hi[d] = zero ? T(0) : f.o[ow];
      lo[d] = zero ? T(0) : f.o[ow - sd];
    }
    if (!IGA) { hi[d] = flux(hi[d], p0, ph[d]); lo[d] = flux(lo[d], pl[d], p0); }
  };
  faces(ic<0>{});
  if constexpr (ND > 1) faces(ic<1>{});
  if constexpr (ND > 2) faces(ic<2>{});
  const int oc = at<ND>(E.bu, c);
  T mn, mx;
  if (MODE == 2) {
    mn = E.mn.o[oc]; mx = E.mx.o[oc];
  } else {
    T l[3], h[3];
#pragma unroll
    for (int d = 0; d < ND; ++d) { l[d] = E.psin.o[ol[d]]; h[d] = E.psin.o[oh[d]]; }
    bounds<ND>(E.psin.o[o0], l, h, mn, mx);
    if (MODE == 1) { E.mn.o[oc] = mn; E.mx.o[oc] = mx; }
  }
  betas<ND>(p0, pl, ph, mn, mx, lo, hi, E.bu.o[oc], E.bd.o[oc]);
}

template <int ND, bool IGA, int MODE, class T>
__global__ void __launch_bounds__(kStageThreads, blocks<T>::betas) k_betas(const __grid_constant__ args<T> A, int nb, int mi) {
  next_may_start();
  const eqn<T> &E = A.e[blockIdx.z];
  if (ND == 1 || int(blockIdx.x) >= nb) {
    int c[3];
    after_previous();
    if (ND == 1 && int(blockIdx.x) < nb) {
      if (own<ND>(A, c)) beta_cell<ND, IGA, MODE>(A, E, c, -1);
      return;
    }
    int d, side;
    if (!face_entry<ND>(A, list_index(nb), 2, d, side, c)) return;
    c[d] = side ? A.n[d] : -1;
    beta_cell<ND, IGA, MODE>(A, E, c, d);
    return;
  }
  if constexpr (ND > 1) {
    walk w;
    if (!column<ND>(A, mi, w)) return;
    const int j = w.j, k = w.k;
    const int o = in_plane<ND>(E.in, j, k), oj = in_plane<ND>(E.in, src(A, 1, j + 1), k), ojm = in_plane<ND>(E.in, src(A, 1, j - 1), k);
    const int ok = ND == 3 ? in_plane<ND>(E.in, j, src(A, 2, k + 1)) : 0, okm = ND == 3 ? in_plane<ND>(E.in, j, src(A, 2, k - 1)) : 0;
    const arr<T> &F0 = E.corr[0], &F1 = E.corr[1], &F2 = E.corr[ND - 1];
    const int a0 = in_plane<ND>(F0, j, k), a1 = in_plane<ND>(F1, j, k), a2 = in_plane<ND>(F2, j, k), s1 = ND == 3 ? F1.s1 : 1;
    auto plane = [&](const arr<T> &f, int i) { return f.o + (long long)i * f.s0; };
    after_previous();
    T p0 = plane(E.in, w.i0)[o], pm = plane(E.in, src(A, 0, w.i0 - 1))[o], c0 = plane(F0, w.i0 - 1)[a0];
    T q0 = T(0), qm = T(0);
    if (MODE != 2) { q0 = plane(E.psin, w.i0)[o]; qm = plane(E.psin, src(A, 0, w.i0 - 1))[o]; }
#pragma unroll 2
    for (int i = w.i0; i < w.i1; ++i) {
      const int ip = src(A, 0, i + 1);
      const auto p = plane(E.in, i), f1 = plane(F1, i);
      const T pn = plane(E.in, ip)[o], c1 = plane(F0, i)[a0];
      T ph[3], pl[3], hi[3], lo[3];
      ph[0] = pn; pl[0] = pm; hi[0] = c1; lo[0] = c0;
      ph[1] = p[oj]; pl[1] = p[ojm]; hi[1] = f1[a1]; lo[1] = f1[a1 - s1];
      if (ND == 3) { const auto f2 = plane(F2, i); ph[2] = p[ok]; pl[2] = p[okm]; hi[2] = f2[a2]; lo[2] = f2[a2 - 1]; }
      const long long oc = (long long)i * E.bu.s0 + o;  // the limiters have the layout of psi
      T mn, mx, qn = T(0);
      if (MODE == 2) {
        mn = E.mn.o[oc]; mx = E.mx.o[oc];
      } else {
        const auto q = plane(E.psin, i);
        qn = plane(E.psin, ip)[o];
        T h[3] = {qn, q[oj], T(0)}, l[3] = {qm, q[ojm], T(0)};
        if (ND == 3) { h[2] = q[ok]; l[2] = q[okm]; }
        bounds<ND>(q0, l, h, mn, mx);
        if (MODE == 1) { E.mn.o[oc] = mn; E.mx.o[oc] = mx; }
      }
      if (!IGA)
#pragma unroll
        for (int d = 0; d < ND; ++d) { hi[d] = flux(hi[d], p0, ph[d]); lo[d] = flux(lo[d], pl[d], p0); }
      betas<ND>(p0, pl, ph, mn, mx, lo, hi, E.bu.o[oc], E.bd.o[oc]);
      c0 = c1; pm = p0; p0 = pn; qm = q0; q0 = qn;
    }
  }
}

// ---- corrective donor-cell pass ----
template <class T>
__device__ __forceinline__ T limited(T C, T bul, T bdl, T bur, T bdr) {  // GC_mono (l: cell below the face, r: above)
  return C * (C > T(0) ? dmin(T(1), dmin(bdl, bur)) : dmin(T(1), dmin(bul, bdr)));
}

template <int ND, bool IGA, bool FCT, class T>
__global__ void __launch_bounds__(kStageThreads, blocks<T>::correct) k_correct(const __grid_constant__ args<T> A, int mi) {
  next_may_start();
  const eqn<T> &E = A.e[blockIdx.z];
  if constexpr (ND == 1) {
    int c[3];
    if (!own<ND>(A, c)) return;
    after_previous();
    const int x = c[0];
    const auto p = E.in.o, f = E.corr[0].o, bu = E.bu.o, bd = E.bd.o;
    T ch = f[x], cl = f[x - 1];
    if (FCT) {
      ch = limited(ch, bu[x], bd[x], bu[x + 1], bd[x + 1]);
      cl = limited(cl, bu[x - 1], bd[x - 1], bu[x], bd[x]);
    }
    const T p0 = p[x], pp = IGA ? T(0) : p[src(A, 0, x + 1)], pm = IGA ? T(0) : p[src(A, 0, x - 1)];
    const T nt = net(A, 0, x, [&](int w) { return IGA ? (w == 0 ? ch : cl) : (w == 0 ? flux(ch, p0, pp) : flux(cl, pm, p0)); });
    E.out.o[x] = p0 + nt;
  } else {
    walk w;
    if (!column<ND>(A, mi, w)) return;
    const int j = w.j, k = w.k;
    const int o = in_plane<ND>(E.in, j, k), oj = in_plane<ND>(E.in, src(A, 1, j + 1), k), ojm = in_plane<ND>(E.in, src(A, 1, j - 1), k);
    const int ok = ND == 3 ? in_plane<ND>(E.in, j, src(A, 2, k + 1)) : 0, okm = ND == 3 ? in_plane<ND>(E.in, j, src(A, 2, k - 1)) : 0;
    const int sj = ND == 3 ? E.in.s1 : 1;  // the limiters have the layout of psi, with their halo cells
    const arr<T> &F0 = E.corr[0], &F1 = E.corr[1], &F2 = E.corr[ND - 1];
    const int a0 = in_plane<ND>(F0, j, k), a1 = in_plane<ND>(F1, j, k), a2 = in_plane<ND>(F2, j, k), s1 = ND == 3 ? F1.s1 : 1;
    auto plane = [&](const arr<T> &f, int i) { return f.o + (long long)i * f.s0; };
    after_previous();
    T p0 = plane(E.in, w.i0)[o], bu0 = T(0), bd0 = T(0), lo = plane(F0, w.i0 - 1)[a0];
    if (FCT) {
      bu0 = plane(E.bu, w.i0)[o]; bd0 = plane(E.bd, w.i0)[o];
      lo = limited(lo, plane(E.bu, w.i0 - 1)[o], plane(E.bd, w.i0 - 1)[o], bu0, bd0);
    }
    if (!IGA) lo = flux(lo, plane(E.in, src(A, 0, w.i0 - 1))[o], p0);
#pragma unroll 2
    for (int i = w.i0; i < w.i1; ++i) {
      const auto q = plane(E.in, i), f1 = plane(F1, i);
      T pn = T(0), bun = T(0), bdn = T(0), hi = plane(F0, i)[a0];
      T yh = f1[a1], yl = f1[a1 - s1];
      if (!IGA || i + 1 < w.i1) pn = plane(E.in, src(A, 0, i + 1))[o];
      if (FCT) {
        const auto u = plane(E.bu, i), v = plane(E.bd, i);
        bun = plane(E.bu, i + 1)[o]; bdn = plane(E.bd, i + 1)[o];
        hi = limited(hi, bu0, bd0, bun, bdn);
        yh = limited(yh, bu0, bd0, u[o + sj], v[o + sj]);
        yl = limited(yl, u[o - sj], v[o - sj], bu0, bd0);
      }
      if (!IGA) { hi = flux(hi, p0, pn); yh = flux(yh, p0, q[oj]); yl = flux(yl, q[ojm], p0); }
      T nt[3];
      nt[0] = net(A, 0, i, [&](int f) { return f == 0 ? hi : lo; });
      nt[1] = net(A, 1, j, [&](int f) { return f == 0 ? yh : yl; });
      if constexpr (ND == 3) {
        const auto f2 = plane(F2, i);
        T zh = f2[a2], zl = f2[a2 - 1];
        if (FCT) {
          const auto u = plane(E.bu, i), v = plane(E.bd, i);
          zh = limited(zh, bu0, bd0, u[o + 1], v[o + 1]);
          zl = limited(zl, u[o - 1], v[o - 1], bu0, bd0);
        }
        if (!IGA) { zh = flux(zh, p0, q[ok]); zl = flux(zl, q[okm], p0); }
        nt[2] = net(A, 2, k, [&](int f) { return f == 0 ? zh : zl; });
      }
      E.out.o[(long long)i * E.out.s0 + o] = donor<ND>(p0, nt);
      lo = hi; p0 = pn; bu0 = bun; bd0 = bdn;
    }
  }
}

// ---- one-dimensional problems: several steps per launch in registers ----
// A warp holds 128 consecutive points, 4 per lane, and takes `steps` steps of its
// segment alone; neighbours come by shuffles.  Every step spoils at most `radius`
// points at each end of the segment, so the outermost steps * radius points are halo:
// computed, not written, and no warp waits for another.  A cyclic axis whose point
// n-1 repeats point 0 is unrolled with period n-1; outside an open axis every stage
// takes the edge values that its halo fill would give it.  Arithmetic of the stages
// above.  Bound by the latency of one step (divisions and shuffles in sequence) and,
// with many segments, by issue.
constexpr int kLinePoints = 128;
// points that one step spoils: psi1 1, then per corrective pass the donor-cell sum 1,
// the limiter 1 and a third-order term 1
__host__ __device__ constexpr int line_radius(int passes, bool fct, bool tot) {
  return 1 + (passes - 1) * (1 + (fct ? 1 : 0) + (tot ? 1 : 0));
}

template <class T>
struct line_args {
  fptr<T> in[kStageEqns], out[kStageEqns];
  fptr<T> gc;  // faces -hv .. n-2+hv
  int n, steps, halo, hv;
  bool cyclic;
  long long t0;
  int uff;
};

template <class T>
struct q4 {
  T v[4];
  __device__ __forceinline__ T operator[](int e) const { return v[e]; }
  __device__ __forceinline__ T &operator[](int e) { return v[e]; }
};
template <class T> __device__ __forceinline__ q4<T> left(const q4<T> &a) {  // values one point below
  return {{__shfl_up_sync(0xffffffffu, a.v[3], 1), a.v[0], a.v[1], a.v[2]}};
}
template <class T> __device__ __forceinline__ q4<T> right(const q4<T> &a) {
  return {{a.v[1], a.v[2], a.v[3], __shfl_down_sync(0xffffffffu, a.v[0], 1)}};
}
#define MPDX_EACH for (int e = 0; e < 4; ++e)

template <int NI, bool FCT, bool IGA, bool TOT, class T>
__global__ void __launch_bounds__(128) k_line(const line_args<T> A) {
  const int lane = threadIdx.x & 31, seg = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int useful = kLinePoints - 2 * A.halo, n = A.n, P = A.cyclic ? n - 1 : n;
  const int x0 = seg * useful;
  if (x0 >= P) return;  // whole warps
  const int xs = x0 - A.halo;  // first point of the segment
  const auto in = A.in[blockIdx.y], out = A.out[blockIdx.y];
  next_may_start();
  after_previous();
  int x[4];
  q4<T> p, C0;
#pragma unroll
  MPDX_EACH {
    x[e] = xs + 4 * lane + e;
    int q = x[e];
    if (A.cyclic) { q %= P; q += q < 0 ? P : 0; }
    p[e] = in[A.cyclic ? q : min(max(q, 0), n - 1)];
    C0[e] = A.gc[A.cyclic ? q : min(max(q, -A.hv), n - 2 + A.hv)];
  }
  // whether the segment reaches outside an open axis
  const bool edge = !A.cyclic && (xs < 0 || xs + kLinePoints > n);
  auto pick = [&](const q4<T> &a, int q) {  // value at point q of the segment
    const int w = q - xs;
    const T u = (w & 3) == 0 ? a[0] : ((w & 3) == 1 ? a[1] : ((w & 3) == 2 ? a[2] : a[3]));
    return __shfl_sync(0xffffffffu, u, (w >> 2) & 31);
  };
  auto fill = [&](q4<T> &a) {  // open scalar fill
    if (!edge) return;
    const T l = pick(a, 0), r = pick(a, n - 1);
#pragma unroll
    MPDX_EACH {
      if (x[e] < 0) a[e] = l;
      if (x[e] > n - 1) a[e] = r;
    }
  };
  auto fill_v = [&](q4<T> &a) {  // open along-axis fill of an antidiffusive velocity (open_1d.hpp)
    if (!edge) return;
    const T l = pick(a, 0), r = pick(a, n - 3);
#pragma unroll
    MPDX_EACH {
      if (x[e] < -1) a[e] = l;
      if (x[e] > n - 1) a[e] = r;
    }
  };
  auto donor_cell = [&](const q4<T> &a, const q4<T> &f) {
    const q4<T> fl = left(f);
    q4<T> r;
#pragma unroll
    MPDX_EACH r[e] = a[e] + (-f[e] + fl[e]);
    return r;
  };
  auto fluxes = [&](const q4<T> &c, const q4<T> &a) {
    const q4<T> ar = right(a);
    q4<T> f;
#pragma unroll
    MPDX_EACH f[e] = flux(c[e], a[e], ar[e]);
    return f;
  };
  for (int s = 0; s < A.steps; ++s) {
    q4<T> mn, mx;
    if (FCT) {
      fill(p);
      const q4<T> l = left(p), r = right(p);
#pragma unroll
      MPDX_EACH {
        mn[e] = dmin(dmin(l[e], p[e]), r[e]);
        mx[e] = dmax(dmax(l[e], p[e]), r[e]);
      }
    } else {
      fill(p);
    }
    p = donor_cell(p, fluxes(C0, p));
    if (NI == 1 || (A.uff > 0 && (A.t0 + s) % A.uff == 0)) continue;
    q4<T> C = C0;
#pragma unroll
    for (int it = 1; it < NI; ++it) {
      fill(p);
      const q4<T> pr = right(p), pl = left(p);
      q4<T> prr = pr;
      if (TOT) prr = right(pr);
#pragma unroll
      MPDX_EACH {
        const T c = C[e], p1 = pr[e], p0 = p[e];
        const T ndx = IGA ? T(2) * (p1 - p0) / T(2) : T(2) * frac(p1 - p0, p1 + p0);
        T r = fabs(c) / T(2) * (T(1) - fabs(c)) * ndx;
        if (TOT) r = r + nd2<IGA>(prr[e], p1, p0, pl[e]) * cxx(c);
        C[e] = r;
      }
      q4<T> f;
      if (FCT) {
        fill_v(C);
        f = C;
        if (!IGA) f = fluxes(C, p);
        const q4<T> fl = left(f);
        q4<T> bu, bd;
#pragma unroll
        MPDX_EACH {
          const T h = dmax(mx[e], dmax(pl[e], dmax(p[e], pr[e]))), l = dmin(mn[e], dmin(pl[e], dmin(p[e], pr[e])));
          const T du = pos(fl[e]) - neg(f[e]), dd = pos(f[e]) - neg(fl[e]);
          bu[e] = (h - p[e]) / (du + lim<T>::eps());
          bd[e] = (p[e] - l) / (dd + lim<T>::eps());
        }
        const q4<T> bur = right(bu), bdr = right(bd);
        q4<T> m;
#pragma unroll
        MPDX_EACH m[e] = C[e] * (C[e] > T(0) ? dmin(T(1), dmin(bd[e], bur[e])) : dmin(T(1), dmin(bu[e], bdr[e])));
        f = m;
        if (!IGA) f = fluxes(m, p);
      } else {
        f = C;
        if (!IGA) f = fluxes(C, p);
      }
      p = donor_cell(p, f);
    }
  }
#pragma unroll
  MPDX_EACH {
    if (x[e] < x0 || x[e] >= min(x0 + useful, P)) continue;
    out[x[e]] = p[e];
    if (A.cyclic && x[e] == 0) out[n - 1] = p[e];
  }
}
#undef MPDX_EACH

template <int NI, bool FCT, class T>
void launch_line(const mpdata_state<T> &st, dim3 g, int bs, const line_args<T> &a) {
  const bool iga = st.opts & o_iga, tot = st.opts & o_tot;
  if (iga && tot) launch_dependent(k_line<NI, FCT, true, true, T>, g, bs, st.stream, a);
  else if (iga) launch_dependent(k_line<NI, FCT, true, false, T>, g, bs, st.stream, a);
  else if (tot) launch_dependent(k_line<NI, FCT, false, true, T>, g, bs, st.stream, a);
  else launch_dependent(k_line<NI, FCT, false, false, T>, g, bs, st.stream, a);
}

// ---- host ----
// Planes that a thread walks: at most 8, halved while fewer than 1100 blocks would run.
// FP64 us per step for 1, 2, 4 and 8 planes: 59^3 fct 36, 39, 47, 69; 97 x 89 x 65
// iga|fct 61, 55, 54, 76; 1024^2 fct in three passes 112, 97, 96, 119;
// 250 x 257 x 241 iga|fct 1419, 1099, 989, 976.
inline int planes_per_thread(int n0, long long blocks) {
  int mi = 8;
  while (mi > 1 && blocks * ceil_div(n0, mi) < 1100) mi /= 2;
  while (ceil_div(n0, mi) > 65535) mi *= 2;  // blocks along the grid's second axis
  return mi;
}

template <class T>
arr<T> view(const field<T> &f) {
  return {pointer(f.v), int(f.v.s0), int(f.v.s1)};
}

template <class T, int ND>
void step_nd(mpdata_state<T> &st, stage_engine<T> &eng, int e0, int ne, int passes) {
  args<T> A;
  for (int d = 0; d < 3; ++d) {
    A.n[d] = st.n[d];
    A.bc[d][0] = st.bcs[d][0];
    A.bc[d][1] = st.bcs[d][1];
  }
  const bool fct = st.opts & o_fct, iga = st.opts & o_iga, tot = st.opts & o_tot;
  const int bs = kStageThreads, pos = ND == 1 ? st.n[0] : (ND == 2 ? st.n[1] : st.n[1] * st.n[2]);
  const int nb = int(ceil_div(pos, bs));
  const int mi = ND == 1 ? 1 : planes_per_thread(st.n[0], (long long)nb * ne);
  const int ny = ND == 1 ? 1 : int(ceil_div(st.n[0], mi));
  const dim3 grid(nb, ny, ne);
  long long faces = 0;  // positions of one face per axis
  for (int d = 0; d < ND; ++d) faces += st.cells() / st.n[d];
  auto with_list = [&](long long entries) { return dim3(nb + ceil_div(entries, (long long)bs * ny), ny, ne); };
  cudaStream_t s = st.stream;
  for (int it = 0; it < passes; ++it) {
    for (int q = 0; q < ne; ++q) {
      eqn<T> &E = A.e[q];
      const int e = e0 + q, tl = st.tl[e];
      typename stage_engine<T>::work *w = q > 0 ? &eng.more[q - 1] : nullptr;
      field<T> *t0 = w ? w->tmp0 : st.tmp0, *t1 = w ? w->tmp1 : st.tmp1;
      E.in = view(st.psi[e][tl ^ (it & 1)]);
      E.out = view(st.psi[e][tl ^ (it & 1) ^ 1]);
      E.psin = view(st.psi[e][tl]);
      for (int d = 0; d < 3; ++d) {
        const int dd = d < ND ? d : 0;
        E.corr[d] = view(it == 2 ? t1[dd] : t0[dd]);
        E.unco[d] = view(it < 2 ? st.GC[dd] : t0[dd]);
      }
      if (fct) {
        E.bu = view(w ? w->beta_up : st.beta_up);
        E.bd = view(w ? w->beta_dn : st.beta_dn);
        E.mn = view(w ? w->psi_min : st.psi_min);
        E.mx = view(w ? w->psi_max : st.psi_max);
      }
    }
    if (it == 0) {
      launch_dependent(k_upwind<ND, T>, grid, bs, s, A, mi);
      continue;
    }
    const dim3 ga = with_list(fct && ND > 1 ? 2 * faces : faces), gb = with_list(2 * faces);
    auto anti = [&](auto ig, auto to) {
      constexpr bool IG = decltype(ig)::value, TO = decltype(to)::value;
      if (it == 1) launch_dependent(k_antidiff<ND, IG, TO, true, T>, ga, bs, s, A, nb, mi, fct);
      else launch_dependent(k_antidiff<ND, IG, TO, false, T>, ga, bs, s, A, nb, mi, fct);
    };
    auto rest = [&](auto ig) {
      constexpr bool IG = decltype(ig)::value;
      if (fct) {
        if (it == 2) launch_dependent(k_betas<ND, IG, 2, T>, gb, bs, s, A, nb, mi);
        else if (passes > 2) launch_dependent(k_betas<ND, IG, 1, T>, gb, bs, s, A, nb, mi);
        else launch_dependent(k_betas<ND, IG, 0, T>, gb, bs, s, A, nb, mi);
        launch_dependent(k_correct<ND, IG, true, T>, grid, bs, s, A, mi);
      } else {
        launch_dependent(k_correct<ND, IG, false, T>, grid, bs, s, A, mi);
      }
    };
    if (iga && tot) anti(std::true_type{}, std::true_type{});
    else if (iga) anti(std::true_type{}, std::false_type{});
    else if (tot) anti(std::false_type{}, std::true_type{});
    else anti(std::false_type{}, std::false_type{});
    if (iga) rest(std::true_type{});
    else rest(std::false_type{});
  }
  if (passes & 1)
    for (int q = 0; q < ne; ++q) st.tl[e0 + q] ^= 1;
}

}  // namespace sg

template <class T>
bool stage_engine<T>::covers(const mpdata_state<T> &st) {
  if (st.opts & ~(o_fct | o_iga | o_tot)) return false;
  if (st.n_iters < 1 || st.n_iters > 3) return false;
  bool rigid = false;
  for (int d = 0; d < st.nd; ++d) {
    if (st.n[d] < 2 * st.H + 1) return false;
    for (int q = 0; q < 2; ++q) rigid = rigid || st.bcs[d][q] == MPDX_BC_RIGID;
    if ((st.bcs[d][0] == MPDX_BC_CYCLIC) != (st.bcs[d][1] == MPDX_BC_CYCLIC)) return false;
  }
  // the reference then rewrites the velocity that the third pass corrects (xchng_flux
  // on the fluxes of the infinite gauge, which are that velocity)
  if (st.n_iters == 3 && (st.opts & o_iga) && !(st.opts & o_fct) && rigid) return false;
  if (st.nd == 3 && st.n[0] > 65535) return false;
  // 32-bit offsets
  size_t most = st.psi[0][0].bytes;
  for (int d = 0; d < st.nd; ++d) most = std::max(most, st.GC[d].bytes);
  return most / sizeof(T) < (size_t(1) << 31) - 65536;
}

template <class T>
bool stage_engine<T>::line_covers(const mpdata_state<T> &st) {
  if (st.nd != 1 || !covers(st)) return false;
  const int l = st.bcs[0][0], r = st.bcs[0][1];
  return (l == MPDX_BC_CYCLIC && r == MPDX_BC_CYCLIC) || (l == MPDX_BC_OPEN && r == MPDX_BC_OPEN);
}

template <class T>
void stage_engine<T>::line(mpdata_state<T> &st, long long nt) {
  const bool fct = st.opts & o_fct, tot = st.opts & o_tot;
  const int radius = sg::line_radius(st.n_iters, fct, tot), n = st.n[0];
  // Steps per launch: a launch costs about as much as 10 steps, so as many as leave a
  // quarter of a segment for results while all segments run at once (one warp per
  // scheduler); with more segments than that the halo's work counts and half of a
  // segment is kept.
  const int most = sg::kLinePoints * 3 / 8 / radius, fewer = std::max(1, sg::kLinePoints / 4 / radius);
  int dev = 0, sms = 148;
  MPDX_CUDA(cudaGetDevice(&dev));
  MPDX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const bool few = (long long)n * st.n_eqns <= 4LL * sms * (sg::kLinePoints - 2 * most * radius);
  const int per = few ? most : fewer;
  while (nt > 0) {
    sg::line_args<T> a;
    a.steps = int(std::min<long long>(nt, per));
    a.halo = (a.steps * radius + 3) / 4 * 4;
    a.n = n;
    a.hv = st.H;
    a.cyclic = st.bcs[0][0] == MPDX_BC_CYCLIC;
    a.gc = pointer(st.GC[0].v);
    a.t0 = st.timestep;
    a.uff = st.upwind_filter_freq;
    const int useful = sg::kLinePoints - 2 * a.halo, bs = few ? 32 : 128;
    const int segs = int(ceil_div(a.cyclic ? n - 1 : n, useful));
    for (int e0 = 0; e0 < st.n_eqns; e0 += kStageEqns) {
      const int ne = std::min(kStageEqns, st.n_eqns - e0);
      for (int q = 0; q < ne; ++q) {
        a.in[q] = pointer(st.psi[e0 + q][st.tl[e0 + q]].v);
        a.out[q] = pointer(st.psi[e0 + q][st.tl[e0 + q] ^ 1].v);
        st.tl[e0 + q] ^= 1;
      }
      const dim3 g(ceil_div(segs, bs / 32), ne);
      if (st.n_iters == 1) sg::launch_line<1, false>(st, g, bs, a);
      else if (st.n_iters == 2 && fct) sg::launch_line<2, true>(st, g, bs, a);
      else if (st.n_iters == 2) sg::launch_line<2, false>(st, g, bs, a);
      else if (fct) sg::launch_line<3, true>(st, g, bs, a);
      else sg::launch_line<3, false>(st, g, bs, a);
    }
    st.timestep += a.steps;
    nt -= a.steps;
  }
}

// One launch takes up to kStageEqns equations of a small grid (their work arrays
// together stay in cache and the launches count), one of a large grid.  Open, iga|fct,
// FP64, four equations, us per step one by one and together: 101^2 62 and 16, 364 x 360
// 52 and 26, 64^3 130 and 85, 512^2 71 and 40; above the line the gain goes on but
// falls (724^2 101 and 82, 80^3 195 and 161, 1024^2 167 and 159) while the further work
// arrays (10 fields per equation in 3D) grow, and no size lost: the line keeps them
// to about 100 MB.
constexpr long long kStageBatchCells = 1 << 18;

// The further work arrays are made by the first step that has a use for them.  A step
// that is being captured cannot allocate, and goes equation by equation if it is the
// first; so does every step where memory is short.
template <class T>
int stage_engine<T>::together(mpdata_state<T> &st) {
  const int most = std::min(kStageEqns, st.n_eqns);
  if (most == 1 || st.cells() > kStageBatchCells || one_by_one) return 1;
  if (more_ready) return most;
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  MPDX_CUDA(cudaStreamIsCapturing(st.stream, &c));
  if (c != cudaStreamCaptureStatusNone) return 1;
  try {
    more.resize(most - 1);
    for (auto &w : more) {
      if (st.n_iters == 1) break;  // an upwind pass has no work arrays
      st.alloc_vctr(w.tmp0);
      if (st.n_iters > 2) st.alloc_vctr(w.tmp1);
      if (st.opts & o_fct)
        for (field<T> *f : {&w.beta_up, &w.beta_dn, &w.psi_min, &w.psi_max}) st.alloc_sclr(*f);
    }
  } catch (const error &) {
    (void)cudaGetLastError();
    more.clear();
    one_by_one = true;
    return 1;
  }
  more_ready = true;
  return most;
}

template <class T>
void stage_engine<T>::step(mpdata_state<T> &st, bool upwind_only) {
  const int passes = upwind_only ? 1 : st.n_iters;
  const int most = together(st);
  for (int e0 = 0; e0 < st.n_eqns; e0 += most) {
    const int ne = std::min(most, st.n_eqns - e0);
    if (st.nd == 1) sg::step_nd<T, 1>(st, *this, e0, ne, passes);
    else if (st.nd == 2) sg::step_nd<T, 2>(st, *this, e0, ne, passes);
    else sg::step_nd<T, 3>(st, *this, e0, ne, passes);
  }
}

}  // namespace mpdx
