// xband.cu -- Mehrotra predictor-corrector interior point for separable convex QPs with banded
// inequality rows, in x-space, with the iterate and the Newton solves in double-double.
//
// The shape: min 1/2 x'diag(q)x + c'x over free x subject to a_r x >= b_r, each row spanning at
// most kd + 1 consecutive columns (the convex-sequence QP: rows (1, -2, 1) on x_r, x_r+1, x_r+2).
// The reference reaches this shape's optimum only through its structured LISWET solvers in long
// double / __float128 (solver/qp/src/qp_interior_point.cpp:892-967 detector, :2378-2826 x-space
// pentadiagonal IPM); its generic QP IPM (:2848-3116) stalls on it, and so do FP64 normal equations:
// near the optimum the row weights z/w span more than 1e25, so Q's contribution to
// K = Q + A' diag(z/w) A vanishes below FP64 rounding of the large entries, and the multipliers z
// (up to ~1e7) leave A'z accurate only to ~1e-9. Here K is assembled, factored (block L D L' in an
// odd-even order) and solved in double-double, and x, z, the residuals b - Ax + w and
// Qx + c - A'z, and the direction's dw = A dx + rp and dz are carried in double-double too; the
// slack w, step lengths, mu and sigma stay FP64.
//
// Newton step (rows normalised to >=, slack w = Ax - b >= 0, multiplier z >= 0, theta = z / w):
//   (Q + A' theta A) dx = -rd - A'(rc / w + theta rp),   rp = Ax - w - b,  rd = Qx + c - A'z
//   dw = A dx + rp,   dz = -rc / w - theta dw
// with rc = w z for the predictor and w z + dw_aff dz_aff - sigma mu for the corrector,
// sigma = (mu_aff / mu)^3, one common step min(1, tau * max step) (Q != 0, qp_interior_point.cpp:3095),
// and the reference QP's residual and gap measures (:2975-2994): p_res = |rp|_inf / max(1, |b|_inf),
// d_res = |rd|_inf / max(1, |c|_inf + |Qx|_inf), gap = w'z / (1 + |objective|).
//
// The whole solve is one launch of one thread-block cluster (16 CTAs where the device can place
// one, 4 up to 1024 columns): the vector passes are spread over all its threads, scalars are folded through distributed
// shared memory, and K is factored and solved by odd-even block reduction (reduce_level below).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "common.cuh"
#include "dd.cuh"
#include "xband.hpp"

namespace cg = cooperative_groups;

namespace sov {
namespace {

constexpr int kXbThreads = 512;   // per CTA
constexpr int kXbCluster = 16;    // CTAs of the cluster (8, the portable size, where 16 cannot be placed)
constexpr int kXbSmallCluster = 4;  // with few columns
constexpr int kXbSmall = 1024;
constexpr int kXbMaxLevels = 32;
constexpr int kXbTop = 320;       // levels of at most this many blocks run in CTA 0 alone

struct XbOut {
  int status, iterations, history_len, failed;
  double p_res, d_res, gap, obj, mu;
  double gap_hist[SOV_HISTORY_MAX], mu_hist[SOV_HISTORY_MAX], obj_hist[SOV_HISTORY_MAX];
  double step_hist[SOV_HISTORY_MAX];
  int it_hist[SOV_HISTORY_MAX];
};

struct XbDev {
  int n, m, max_iter;
  const int *row_ptr, *col_idx, *col_ptr, *row_idx;
  const double *row_val, *col_val, *q, *c, *b;
  double obj_constant, bnorm, cnorm, feas_tol, opt_tol, tau;
  // iterates: x and z in double-double, w in FP64
  double *xh, *xl, *zh, *zl, *w;
  // work
  double *th, *rph, *rpl, *rd, *rcw, *uh, *ul, *dxh, *dxl, *dw, *dzh, *dzl, *dwa, *dza;
  // odd-even reduction: per level its block count and first slot; every array below is component
  // major (component c of block i of level l at c * slots + off[l] + i), hi then lo parts
  int levels, natural;
  int size[kXbMaxLevels], off[kXbMaxLevels];
  long long slots;
  double *Dh, *Dl;  // diagonal blocks, lower triangle packed (r (r + 1) / 2 + c)
  double *Bh, *Bl;  // block (i, i - 1), r * kd + c
  double *Fh, *Fl;  // right-hand sides, kd
  double *Lh, *Ll;  // eliminated blocks: unit lower factor (strict, r (r - 1) / 2 + c),
  double *Ih, *Il;  //   1 / D,
  double *Xh, *Xl;  //   X = L^-1 B_o (coupling to the left neighbour), r * kd + c,
  double *Uh, *Ul;  //   U = L^-1 B_{o+1}' (coupling to the right neighbour),
  double *Vh, *Vl;  //   X / D by rows,
  double *Wh, *Wl;  //   U / D by rows,
  double *Qh, *Ql;  //   L^-1 r_o, kd
  int* bad;         // set on a pivot that is not positive and finite
  XbOut* out;
};

__device__ __forceinline__ dd ld_dd(const double* h, const double* l, long long i) { return dd{h[i], l[i]}; }
__device__ __forceinline__ void st_dd(double* h, double* l, long long i, dd v) {
  h[i] = v.hi;
  l[i] = v.lo;
}

// ---- odd-even block reduction ----
// Cut into blocks of KD columns, K is block tridiagonal. A level eliminates its odd blocks: with
// D_o = L diag(d) L' (KD x KD), X = L^-1 B_o and U = L^-1 B_{o+1}' the even neighbours get
//   D_e -= U'd^-1 U (from the left odd block) + X'd^-1 X (from the right one),
//   B_new = -U'd^-1 X,   r_e -= U'd^-1 q + X'd^-1 q,   q = L^-1 r_o,
// and form the next level, half as long; the last level is one block. Back down,
//   x_o = L'^-1 d^-1 (q - X x_{o-1} - U x_{o+1}).
// This is the block L D L' of K in an odd-even (nested dissection) order, with the blocks factored
// rather than inverted: as stable as the natural order (d.natural = 1, SOVEREIGN_XBAND_SEGMENTS=1,
// runs that one on one thread; there is no other number of segments to choose). About 14 levels at n = 20002 replace chains of hundreds of
// dependent double-double steps: what bounds a solve is the latency of one step per level.
// A level is two steps: one thread per odd block factors it and solves for X and U (factor_odd),
// then one thread per entry of the next level's blocks and right-hand sides forms it from both
// neighbours (update_even): the arithmetic of a level, about 1100 FP64 instructions per pair of
// blocks, is spread over all threads and its dependent chain is a few double-double operations.
// Levels are separated by cluster barriers until kXbTop blocks are left; the rest runs in CTA 0.
// Measured on the device (n = 20002, 81 iterations): one CTA with 512 segments and a serial
// separator chain 300 ms; one thread per even block doing a whole level 20.3 ms; this form 17.0 ms.
template <int KD>
__device__ __forceinline__ void load_sym(const XbDev& d, long long at, dd (&A)[KD][KD]) {
#pragma unroll
  for (int r = 0; r < KD; ++r)
#pragma unroll
    for (int c = 0; c <= r; ++c) A[r][c] = ld_dd(d.Dh, d.Dl, (r * (r + 1) / 2 + c) * d.slots + at);
}

template <int KD>
__device__ __forceinline__ void load_full(const double* h, const double* l, long long slots, long long at,
                                          dd (&A)[KD][KD]) {
#pragma unroll
  for (int r = 0; r < KD; ++r)
#pragma unroll
    for (int c = 0; c < KD; ++c) A[r][c] = ld_dd(h, l, (r * KD + c) * slots + at);
}

template <int KD>
__device__ __forceinline__ void store_full(double* h, double* l, long long slots, long long at, const dd (&A)[KD][KD]) {
#pragma unroll
  for (int r = 0; r < KD; ++r)
#pragma unroll
    for (int c = 0; c < KD; ++c) st_dd(h, l, (r * KD + c) * slots + at, A[r][c]);
}

// A (lower triangle) -> unit lower L below the diagonal, 1 / d in inv; false on a pivot that is not
// positive and finite (K = Q + A' theta A is positive definite: only a breakdown gives one)
template <int KD>
__device__ __forceinline__ bool block_ldl(dd (&A)[KD][KD], dd (&inv)[KD]) {
  bool ok = true;
#pragma unroll
  for (int k = 0; k < KD; ++k) {
    const dd p = A[k][k];
    ok = ok && p.hi > 0.0 && isfinite(p.hi);
    inv[k] = dd_recip(p);
    dd lk[KD];
#pragma unroll
    for (int r = k + 1; r < KD; ++r) lk[r] = dd_mul(A[r][k], inv[k]);
#pragma unroll
    for (int r = k + 1; r < KD; ++r) {
#pragma unroll
      for (int c = k + 1; c <= r; ++c) A[r][c] = dd_sub(A[r][c], dd_mul(lk[r], A[c][k]));
    }
#pragma unroll
    for (int r = k + 1; r < KD; ++r) A[r][k] = lk[r];
  }
  return ok;
}

// columns of M <- L^-1 M (L unit lower in A)
template <int KD>
__device__ __forceinline__ void lower_solve(const dd (&A)[KD][KD], dd (&M)[KD][KD]) {
#pragma unroll
  for (int r = 1; r < KD; ++r)
#pragma unroll
    for (int k = 0; k < r; ++k)
#pragma unroll
      for (int c = 0; c < KD; ++c) M[r][c] = dd_sub(M[r][c], dd_mul(A[r][k], M[k][c]));
}
template <int KD>
__device__ __forceinline__ void lower_solve(const dd (&A)[KD][KD], dd (&v)[KD]) {
#pragma unroll
  for (int r = 1; r < KD; ++r)
#pragma unroll
    for (int k = 0; k < r; ++k) v[r] = dd_sub(v[r], dd_mul(A[r][k], v[k]));
}

// row k of M times inv[k]
template <int KD>
__device__ __forceinline__ void scale_rows(dd (&M)[KD][KD], const dd (&inv)[KD]) {
#pragma unroll
  for (int k = 0; k < KD; ++k)
#pragma unroll
    for (int c = 0; c < KD; ++c) M[k][c] = dd_mul(M[k][c], inv[k]);
}

template <int KD>
__device__ __forceinline__ void load_rhs(const double* h, const double* l, long long slots, long long at, dd (&v)[KD]) {
#pragma unroll
  for (int k = 0; k < KD; ++k) v[k] = ld_dd(h, l, k * slots + at);
}
template <int KD>
__device__ __forceinline__ void store_rhs(double* h, double* l, long long slots, long long at, const dd (&v)[KD]) {
#pragma unroll
  for (int k = 0; k < KD; ++k) st_dd(h, l, k * slots + at, v[k]);
}

// The odd blocks of level l: factor, X and U, q = L^-1 r, one thread per block.
template <int KD>
__device__ void factor_odd(const XbDev& d, int l, int t, int threads) {
  const int N = d.size[l];
  const long long S = d.slots;
  for (int h = t; h < N / 2; h += threads) {
    const int i = 2 * h + 1;
    const long long at = d.off[l] + i;
    dd A[KD][KD], M[KD][KD], inv[KD], q[KD];
    load_sym<KD>(d, at, A);
    load_rhs<KD>(d.Fh, d.Fl, S, at, q);
    load_full<KD>(d.Bh, d.Bl, S, at, M);
    if (!block_ldl<KD>(A, inv)) atomicExch(d.bad, 1);
    store_rhs<KD>(d.Ih, d.Il, S, at, inv);
#pragma unroll
    for (int a = 1; a < KD; ++a)
#pragma unroll
      for (int b = 0; b < a; ++b) st_dd(d.Lh, d.Ll, (a * (a - 1) / 2 + b) * S + at, A[a][b]);
    lower_solve<KD>(A, q);
    store_rhs<KD>(d.Qh, d.Ql, S, at, q);
    lower_solve<KD>(A, M);
    store_full<KD>(d.Xh, d.Xl, S, at, M);
    scale_rows<KD>(M, inv);
    store_full<KD>(d.Vh, d.Vl, S, at, M);
    if (i + 1 < N) {
#pragma unroll
      for (int a = 0; a < KD; ++a)
#pragma unroll
        for (int b = 0; b < KD; ++b) M[a][b] = ld_dd(d.Bh, d.Bl, (b * KD + a) * S + at + 1);
      lower_solve<KD>(A, M);
      store_full<KD>(d.Uh, d.Ul, S, at, M);
      scale_rows<KD>(M, inv);
      store_full<KD>(d.Wh, d.Wl, S, at, M);
    }
  }
}

// acc -= sum_k P[k][a] Q[k][b] of block `at` (Q a kd x kd block of `ld` columns, or a vector)
template <int KD>
__device__ __forceinline__ dd minus_product(dd acc, const double* Ph, const double* Pl, int a, const double* Qh,
                                            const double* Ql, int ld, int b, long long S, long long at) {
#pragma unroll
  for (int k = 0; k < KD; ++k)
    acc = dd_sub(acc, dd_mul(ld_dd(Ph, Pl, (k * KD + a) * S + at), ld_dd(Qh, Ql, (k * ld + b) * S + at)));
  return acc;
}

// Level l + 1 from level l's odd blocks, one thread per entry: D_e (lower triangle), r_e, and the
// coupling of an even block to the one before it.
template <int KD>
__device__ void update_even(const XbDev& d, int l, int t, int threads) {
  constexpr int kTri = KD * (KD + 1) / 2, kEntries = kTri + KD + KD * KD;
  const int N = d.size[l], Nn = d.size[l + 1];
  const long long S = d.slots, o0 = d.off[l], o1 = d.off[l + 1];
  for (int u = t; u < kEntries * Nn; u += threads) {
    const int entry = u / Nn, h = u - entry * Nn;
    const long long e = o0 + 2 * h;
    const bool left = h > 0, right = 2 * h + 1 < N;
    if (entry < kTri) {
      int a = 0;
      while ((a + 1) * (a + 2) / 2 <= entry) ++a;
      const int b = entry - a * (a + 1) / 2;
      dd v = ld_dd(d.Dh, d.Dl, entry * S + e);
      if (left) v = minus_product<KD>(v, d.Wh, d.Wl, a, d.Uh, d.Ul, KD, b, S, e - 1);
      if (right) v = minus_product<KD>(v, d.Vh, d.Vl, a, d.Xh, d.Xl, KD, b, S, e + 1);
      st_dd(d.Dh, d.Dl, entry * S + o1 + h, v);
    } else if (entry < kTri + KD) {
      const int a = entry - kTri;
      dd v = ld_dd(d.Fh, d.Fl, a * S + e);
      if (left) v = minus_product<KD>(v, d.Wh, d.Wl, a, d.Qh, d.Ql, 1, 0, S, e - 1);
      if (right) v = minus_product<KD>(v, d.Vh, d.Vl, a, d.Qh, d.Ql, 1, 0, S, e + 1);
      st_dd(d.Fh, d.Fl, a * S + o1 + h, v);
    } else if (left) {
      const int c = entry - kTri - KD, a = c / KD, b = c - a * KD;
      const dd v = minus_product<KD>(dd_from(0.0), d.Wh, d.Wl, a, d.Xh, d.Xl, KD, b, S, e - 1);
      st_dd(d.Bh, d.Bl, c * S + o1 + h, v);
    }
  }
}

template <int KD>
__device__ __forceinline__ void load_lower(const XbDev& d, long long at, dd (&A)[KD][KD]) {
#pragma unroll
  for (int a = 1; a < KD; ++a)
#pragma unroll
    for (int b = 0; b < a; ++b) A[a][b] = ld_dd(d.Lh, d.Ll, (a * (a - 1) / 2 + b) * d.slots + at);
}

// The right-hand side alone down one level, with the factor factor_odd left: one thread per entry
// (q of the odd neighbours, a few operations, is formed by each of them rather than in a step of its own).
template <int KD>
__device__ void forward_level(const XbDev& d, int l, int t, int threads) {
  const int N = d.size[l], Nn = d.size[l + 1];
  const long long S = d.slots, o0 = d.off[l], o1 = d.off[l + 1];
  for (int u = t; u < KD * Nn; u += threads) {
    const int a = u / Nn, h = u - a * Nn;
    const long long e = o0 + 2 * h;
    dd v = ld_dd(d.Fh, d.Fl, a * S + e), q[KD], A[KD][KD];
    if (h > 0) {
      load_rhs<KD>(d.Fh, d.Fl, S, e - 1, q);
      load_lower<KD>(d, e - 1, A);
      lower_solve<KD>(A, q);
#pragma unroll
      for (int k = 0; k < KD; ++k) v = dd_sub(v, dd_mul(ld_dd(d.Wh, d.Wl, (k * KD + a) * S + e - 1), q[k]));
    }
    if (2 * h + 1 < N) {
      load_rhs<KD>(d.Fh, d.Fl, S, e + 1, q);
      load_lower<KD>(d, e + 1, A);
      lower_solve<KD>(A, q);
#pragma unroll
      for (int k = 0; k < KD; ++k) v = dd_sub(v, dd_mul(ld_dd(d.Vh, d.Vl, (k * KD + a) * S + e + 1), q[k]));
      if (a == 0) store_rhs<KD>(d.Qh, d.Ql, S, e + 1, q);
    }
    st_dd(d.Fh, d.Fl, a * S + o1 + h, v);
  }
}

// v <- L'^-1 diag(inv) v
template <int KD>
__device__ __forceinline__ void upper_solve(const dd (&A)[KD][KD], const dd (&inv)[KD], dd (&v)[KD]) {
#pragma unroll
  for (int k = KD - 1; k >= 0; --k) {
    v[k] = dd_mul(v[k], inv[k]);
#pragma unroll
    for (int a = k + 1; a < KD; ++a) v[k] = dd_sub(v[k], dd_mul(A[a][k], v[a]));
  }
}

// The odd blocks of level l from their even neighbours; block i of level l is block i << l of the
// matrix, and solutions go straight to their place in dx. A group of lanes takes a block: lane k
// forms entry k of q - X x_left - U x_right, then all lanes of the group run the small L' solve.
template <int KD>
__device__ void backward_level(const XbDev& d, int l, int t, int threads) {
  constexpr int kLanes = KD <= 2 ? KD : 4;
  const int N = d.size[l], odd = N / 2;
  const long long S = d.slots, o0 = d.off[l];
  const int lane = t % kLanes, k = lane < KD ? lane : KD - 1;
  // whole warps stay in the loop together: the group exchanges its entries by shuffles
  const int warp0 = t & ~31;
  for (int base = warp0 / kLanes; base < odd; base += threads / kLanes) {
    const int h = base + (t - warp0) / kLanes;
    const int i = 2 * min(h, odd - 1) + 1;
    const long long at = o0 + i;
    dd v = ld_dd(d.Qh, d.Ql, k * S + at);
    const long long c0 = static_cast<long long>(i - 1) * KD << l;
#pragma unroll
    for (int c = 0; c < KD; ++c) v = dd_sub(v, dd_mul(ld_dd(d.Xh, d.Xl, (k * KD + c) * S + at), ld_dd(d.dxh, d.dxl, c0 + c)));
    if (i + 1 < N) {
      const long long c1 = static_cast<long long>(i + 1) * KD << l;
#pragma unroll
      for (int c = 0; c < KD; ++c) v = dd_sub(v, dd_mul(ld_dd(d.Uh, d.Ul, (k * KD + c) * S + at), ld_dd(d.dxh, d.dxl, c1 + c)));
    }
    dd x[KD], inv[KD], A[KD][KD];
#pragma unroll
    for (int j = 0; j < KD; ++j) {
      x[j].hi = __shfl_sync(kFull, v.hi, j, kLanes);
      x[j].lo = __shfl_sync(kFull, v.lo, j, kLanes);
    }
    load_rhs<KD>(d.Ih, d.Il, S, at, inv);
    load_lower<KD>(d, at, A);
    upper_solve<KD>(A, inv, x);
    if (h < odd && lane == 0) {
      const long long ci = static_cast<long long>(i) * KD << l;
#pragma unroll
      for (int j = 0; j < KD; ++j) st_dd(d.dxh, d.dxl, ci + j, x[j]);
    }
  }
}

// The one block of the last level.
template <int KD>
__device__ void solve_last(const XbDev& d, bool factor) {
  const long long at = d.off[d.levels - 1];
  dd A[KD][KD], inv[KD], v[KD];
  load_rhs<KD>(d.Fh, d.Fl, d.slots, at, v);
  if (factor) {
    load_sym<KD>(d, at, A);
    if (!block_ldl<KD>(A, inv)) atomicExch(d.bad, 1);
    store_rhs<KD>(d.Ih, d.Il, d.slots, at, inv);
#pragma unroll
    for (int a = 1; a < KD; ++a)
#pragma unroll
      for (int b = 0; b < a; ++b) st_dd(d.Lh, d.Ll, (a * (a - 1) / 2 + b) * d.slots + at, A[a][b]);
  } else {
    load_lower<KD>(d, at, A);
    load_rhs<KD>(d.Ih, d.Il, d.slots, at, inv);
  }
  lower_solve<KD>(A, v);
  upper_solve<KD>(A, inv, v);
#pragma unroll
  for (int k = 0; k < KD; ++k) st_dd(d.dxh, d.dxl, k, v[k]);
}

// The natural order on one thread: block i eliminated into block i + 1.
template <int KD>
__device__ void solve_natural(const XbDev& d, bool factor) {
  const int N = d.size[0];
  const long long S = d.slots;
  dd r[KD], D[KD][KD];
  load_rhs<KD>(d.Fh, d.Fl, S, 0, r);
  if (factor) load_sym<KD>(d, 0, D);
  for (int i = 0; i < N; ++i) {
    dd M[KD][KD], inv[KD], q[KD], A[KD][KD];
#pragma unroll
    for (int k = 0; k < KD; ++k) q[k] = r[k];
    if (factor) {
#pragma unroll
      for (int a = 0; a < KD; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b) A[a][b] = D[a][b];
      if (!block_ldl<KD>(A, inv)) atomicExch(d.bad, 1);
      store_rhs<KD>(d.Ih, d.Il, S, i, inv);
#pragma unroll
      for (int a = 1; a < KD; ++a)
#pragma unroll
        for (int b = 0; b < a; ++b) st_dd(d.Lh, d.Ll, (a * (a - 1) / 2 + b) * S + i, A[a][b]);
    } else {
      load_lower<KD>(d, i, A);
    }
    lower_solve<KD>(A, q);
    store_rhs<KD>(d.Qh, d.Ql, S, i, q);
    if (i + 1 == N) break;
    load_rhs<KD>(d.Fh, d.Fl, S, i + 1, r);
    if (factor) {
      load_sym<KD>(d, i + 1, D);
#pragma unroll
      for (int a = 0; a < KD; ++a)
#pragma unroll
        for (int b = 0; b < KD; ++b) M[a][b] = ld_dd(d.Bh, d.Bl, (b * KD + a) * S + i + 1);
      lower_solve<KD>(A, M);
      store_full<KD>(d.Uh, d.Ul, S, i, M);
#pragma unroll
      for (int k = 0; k < KD; ++k)
#pragma unroll
        for (int a = 0; a < KD; ++a) {
          const dd w = dd_mul(M[k][a], inv[k]);
#pragma unroll
          for (int b = 0; b <= a; ++b) D[a][b] = dd_sub(D[a][b], dd_mul(w, M[k][b]));
          st_dd(d.Wh, d.Wl, (k * KD + a) * S + i, w);
        }
    }
#pragma unroll
    for (int a = 0; a < KD; ++a)
#pragma unroll
      for (int k = 0; k < KD; ++k) r[a] = dd_sub(r[a], dd_mul(ld_dd(d.Wh, d.Wl, (k * KD + a) * S + i), q[k]));
  }
  dd x[KD];
  for (int i = N - 1; i >= 0; --i) {
    dd v[KD], inv[KD], A[KD][KD];
    load_rhs<KD>(d.Qh, d.Ql, S, i, v);
    load_rhs<KD>(d.Ih, d.Il, S, i, inv);
    load_lower<KD>(d, i, A);
    if (i + 1 < N)
#pragma unroll
      for (int c = 0; c < KD; ++c)
#pragma unroll
        for (int k = 0; k < KD; ++k) v[k] = dd_sub(v[k], dd_mul(ld_dd(d.Uh, d.Ul, (k * KD + c) * S + i), x[c]));
    upper_solve<KD>(A, inv, v);
#pragma unroll
    for (int k = 0; k < KD; ++k) {
      x[k] = v[k];
      st_dd(d.dxh, d.dxl, static_cast<long long>(i) * KD + k, v[k]);
    }
  }
}

// K dx = r with r in level 0 of F: with `factor`, K (level 0 of D and B) is factored on the way
// down, else the factor of the last such call is used. Called by the whole cluster after a barrier;
// ends with one.
template <int KD>
__device__ void band_newton(const XbDev& d, bool factor, int t, int threads) {
  cg::cluster_group cluster = cg::this_cluster();
  if (d.natural) {
    if (t == 0) solve_natural<KD>(d, factor);
    cluster.sync();
    return;
  }
  int l = 0;
  for (; d.size[l] > kXbTop; ++l) {
    if (factor) {
      factor_odd<KD>(d, l, t, threads);
      cluster.sync();
      update_even<KD>(d, l, t, threads);
    } else {
      forward_level<KD>(d, l, t, threads);
    }
    cluster.sync();
  }
  if (cluster.block_rank() == 0) {
    const int tt = threadIdx.x;
    int u = l;
    for (; u + 1 < d.levels; ++u) {
      if (factor) {
        factor_odd<KD>(d, u, tt, kXbThreads);
        __syncthreads();
        update_even<KD>(d, u, tt, kXbThreads);
      } else {
        forward_level<KD>(d, u, tt, kXbThreads);
      }
      __syncthreads();
    }
    if (tt == 0) solve_last<KD>(d, factor);
    __syncthreads();
    for (--u; u >= l; --u) {
      backward_level<KD>(d, u, tt, kXbThreads);
      __syncthreads();
    }
  }
  cluster.sync();
  for (--l; l >= 0; --l) {
    backward_level<KD>(d, l, t, threads);
    cluster.sync();
  }
}

// (A v)_r in double-double
__device__ __forceinline__ dd row_dot(const XbDev& d, int r, const double* vh, const double* vl) {
  dd s = dd_from(0.0);
  for (int e = d.row_ptr[r]; e < d.row_ptr[r + 1]; ++e) s = dd_add(s, dd_mul_d(ld_dd(vh, vl, d.col_idx[e]), d.row_val[e]));
  return s;
}

// (A' u)_j in double-double
__device__ __forceinline__ dd col_dot(const XbDev& d, int j, const double* uh, const double* ul) {
  dd s = dd_from(0.0);
  for (int e = d.col_ptr[j]; e < d.col_ptr[j + 1]; ++e) s = dd_add(s, dd_mul_d(ld_dd(uh, ul, d.row_idx[e]), d.col_val[e]));
  return s;
}

// Cluster-wide reduction of NV values (ops: 0 sum, 1 max, 2 min): every CTA's result is written to
// all CTAs' shared memory, and after one cluster barrier every thread folds them in rank order.
// Two buffers taken in turn: a buffer is written again only after a later barrier.
struct ClusterRed {
  double v[2][5][kXbCluster];
};
template <int NV>
__device__ __forceinline__ void cluster_reduce(double (&v)[NV], const int (&ops)[NV], double* red, ClusterRed& cr,
                                               int& turn) {
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = cluster.num_blocks();
  block_reduce<NV>(v, ops, red);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) red[k] = v[k];
  __syncthreads();
  if (static_cast<int>(threadIdx.x) < ctas) {
    ClusterRed* other = cluster.map_shared_rank(&cr, threadIdx.x);
#pragma unroll
    for (int k = 0; k < NV; ++k) other->v[turn][k][cluster.block_rank()] = red[k];
  }
  cluster.sync();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double acc = cr.v[turn][k][0];
    for (int c = 1; c < ctas; ++c) {
      const double u = cr.v[turn][k][c];
      acc = ops[k] == 0 ? acc + u : ops[k] == 1 ? fmax(acc, u) : fmin(acc, u);
    }
    v[k] = acc;
  }
  turn ^= 1;
}

template <int KD>
__global__ void __launch_bounds__(kXbThreads, 1) k_xband_ipm(const __grid_constant__ XbDev d) {
  __shared__ double red[5 * 32];
  __shared__ ClusterRed cr;
  cg::cluster_group cluster = cg::this_cluster();
  int turn = 0;
  const int threads = static_cast<int>(cluster.num_blocks()) * kXbThreads;
  // warps numbered across the CTAs, so that a level with fewer blocks than threads uses every SM
  const int tid = static_cast<int>((threadIdx.x >> 5) * cluster.num_blocks() + cluster.block_rank()) * 32 +
                  static_cast<int>(threadIdx.x & 31);
  const int n = d.n, m = d.m;
  const double inf = INFINITY;
  // the reference QP stops at its tolerances; this path goes two decades further (cheap in
  // double-double) so that its objective meets the exact structured answer to 1e-8
  const double ftol = d.feas_tol * 1e-2, otol = d.opt_tol * 1e-2;
  // every CTA runs (its shared memory can be written) before the first remote store
  cluster.sync();
  int it = 0;
  for (;; ++it) {
    // ---- residuals, mu, objective; theta and the predictor's u = rc / w + theta rp ----
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // max |rp|, max |rd|, max |Qx|, w'z, objective
    for (int r = tid; r < m; r += threads) {
      const double w = d.w[r], z = d.zh[r], th = z / w;
      const dd rp = dd_add_d(dd_add_d(row_dot(d, r, d.xh, d.xl), -w), -d.b[r]);
      st_dd(d.rph, d.rpl, r, rp);
      // rc / w is FP64: the direction has to take this very value again, or its error (1e-16 of z,
      // which reaches 1e7) stays in the dual residual
      const double q = w * z / w;
      d.th[r] = th;
      d.rcw[r] = q;
      st_dd(d.uh, d.ul, r, dd_add_d(dd_mul_d(rp, th), q));
      v[0] = fmax(v[0], fabs(rp.hi));
      v[3] += w * z;
    }
    for (int j = tid; j < n; j += threads) {
      const dd qx = dd_mul_d(ld_dd(d.xh, d.xl, j), d.q[j]);
      const dd rd = dd_sub(dd_add_d(qx, d.c[j]), col_dot(d, j, d.zh, d.zl));
      d.rd[j] = rd.hi;
      v[1] = fmax(v[1], fabs(rd.hi));
      v[2] = fmax(v[2], fabs(qx.hi));
      v[4] += d.c[j] * d.xh[j] + 0.5 * d.q[j] * d.xh[j] * d.xh[j];
    }
    const int ops5[5] = {1, 1, 1, 0, 0}, ops1[1] = {0};
    cluster_reduce<5>(v, ops5, red, cr, turn);
    // every thread holds the same sums, so the whole cluster takes the same decision
    const double mu = v[3] / m;
    const double obj = v[4] + d.obj_constant;
    const double p_res = v[0] / d.bnorm;
    const double d_res = v[1] / fmax(1.0, d.cnorm + v[2]);
    const double gap = v[3] / (1.0 + fabs(obj));
    int status = -1, failed = 0;
    if (!isfinite(mu) || !isfinite(p_res) || !isfinite(d_res)) {
      status = SOV_ERROR;
      failed = 1;
    } else if (p_res <= ftol && d_res <= ftol && gap <= otol) {
      status = SOV_OPTIMAL;
    } else if (it >= d.max_iter) {
      // at the limit the reference QP's own tolerances decide; otherwise ERROR without an
      // objective, as its failure exits publish (qp_interior_point.cpp:3042-3048, :3112-3115)
      status = (p_res <= d.feas_tol && d_res <= d.feas_tol && gap <= d.opt_tol) ? SOV_OPTIMAL : SOV_ERROR;
    }
    if (tid == 0) {
      XbOut* o = d.out;
      o->p_res = p_res;
      o->d_res = d_res;
      o->gap = gap;
      o->obj = obj;
      o->mu = mu;
      o->iterations = it;
      if (o->history_len < SOV_HISTORY_MAX) {
        const int h = o->history_len++;
        o->it_hist[h] = it;
        o->gap_hist[h] = gap;
        o->mu_hist[h] = mu;
        o->obj_hist[h] = obj;
      }
      if (status >= 0) {
        o->status = status;
        o->failed = failed;
      }
    }
    if (status >= 0) break;
    // ---- K = Q + A' theta A in double-double into level 0's blocks, predictor's rhs = -rd - A'u ----
    for (int j = tid; j < d.size[0] * KD; j += threads) {
      const int blk = j / KD, jr = j - blk * KD;
      dd acc[KD + 1];
#pragma unroll
      for (int p = 0; p <= KD; ++p) acc[p] = dd_from(0.0);
      dd rhs = dd_from(0.0);
      if (j < n) {
        acc[0] = dd_from(d.q[j]);
        dd au = dd_from(0.0);
        for (int e = d.col_ptr[j]; e < d.col_ptr[j + 1]; ++e) {
          const int r = d.row_idx[e];
          const double a = d.col_val[e], t = d.th[r];
          au = dd_add(au, dd_mul_d(ld_dd(d.uh, d.ul, r), a));
          for (int f = d.row_ptr[r]; f < d.row_ptr[r + 1]; ++f) {
            const int k = d.col_idx[f];
            const int p = j - k;
            if (p < 0 || p > KD) continue;
            const dd prod = dd_mul_d(two_prod(a, d.row_val[f]), t);
#pragma unroll
            for (int q = 0; q <= KD; ++q)
              if (q == p) acc[q] = dd_add(acc[q], prod);
          }
        }
        rhs = dd_neg(dd_add_d(au, d.rd[j]));
      } else {
        acc[0] = dd_from(1.0);  // columns that pad the last block: an identity
      }
      // K(j, j - p): column jr - p of this block's diagonal, or KD + jr - p of the block before
#pragma unroll
      for (int p = 0; p <= KD; ++p)
        if (p <= jr) st_dd(d.Dh, d.Dl, (jr * (jr + 1) / 2 + jr - p) * d.slots + blk, acc[p]);
        else st_dd(d.Bh, d.Bl, (jr * KD + KD + jr - p) * d.slots + blk, acc[p]);
      for (int c = 0; c < jr; ++c) st_dd(d.Bh, d.Bl, (jr * KD + c) * d.slots + blk, dd_from(0.0));
      st_dd(d.Fh, d.Fl, jr * d.slots + blk, rhs);
    }
    cluster.sync();
    // ---- predictor (pass 0) and corrector (pass 1) ----
    double alpha_p = 1.0, alpha_d = 1.0;
    bool bad = false;
    for (int pass = 0; pass < 2; ++pass) {
      double sigma_mu = 0.0;
      if (pass == 1) {
        // mu_aff and sigma = (mu_aff / mu)^3 (qp_interior_point.cpp, as interior_point.cpp:666-673)
        double ma[1] = {0.0};
        for (int r = tid; r < m; r += threads) {
          d.dwa[r] = d.dw[r];
          d.dza[r] = d.dzh[r];
          ma[0] += (d.w[r] + alpha_p * d.dw[r]) * (d.zh[r] + alpha_d * d.dzh[r]);
        }
        cluster_reduce<1>(ma, ops1, red, cr, turn);
        const double ratio = (ma[0] / m) / mu;
        sigma_mu = fmin(1.0, ratio * ratio * ratio) * mu;
        for (int r = tid; r < m; r += threads) {
          const double q = (d.w[r] * d.zh[r] + d.dwa[r] * d.dza[r] - sigma_mu) / d.w[r];
          d.rcw[r] = q;
          st_dd(d.uh, d.ul, r, dd_add_d(dd_mul_d(ld_dd(d.rph, d.rpl, r), d.th[r]), q));
        }
        cluster.sync();
        for (int j = tid; j < d.size[0] * KD; j += threads) {
          const int blk = j / KD, jr = j - blk * KD;
          st_dd(d.Fh, d.Fl, jr * d.slots + blk,
                j < n ? dd_neg(dd_add_d(col_dot(d, j, d.uh, d.ul), d.rd[j])) : dd_from(0.0));
        }
        cluster.sync();
      }
      band_newton<KD>(d, pass == 0, tid, threads);
      if (pass == 0) {
        bad = *static_cast<volatile int*>(d.bad) != 0;  // every block has its pivots by now
        if (bad) break;
      }
      // dw = A dx + rp, dz = -rc / w - theta dw; largest steps to the boundary
      double a[2] = {inf, inf};
      for (int r = tid; r < m; r += threads) {
        const dd dwv = dd_add(row_dot(d, r, d.dxh, d.dxl), ld_dd(d.rph, d.rpl, r));
        const dd dzv = dd_neg(dd_add_d(dd_mul_d(dwv, d.th[r]), d.rcw[r]));
        d.dw[r] = dwv.hi;
        st_dd(d.dzh, d.dzl, r, dzv);
        if (dwv.hi < 0.0) a[0] = fmin(a[0], -d.w[r] / dwv.hi);
        if (dzv.hi < 0.0) a[1] = fmin(a[1], -d.zh[r] / dzv.hi);
      }
      const int ops2[2] = {2, 2};
      cluster_reduce<2>(a, ops2, red, cr, turn);
      alpha_p = fmin(1.0, a[0]);
      alpha_d = fmin(1.0, a[1]);
    }
    if (bad) {
      if (tid == 0) {
        d.out->status = SOV_ERROR;
        d.out->failed = 2;
      }
      break;
    }
    // ---- common step ----
    const double alpha = fmin(1.0, d.tau * fmin(alpha_p, alpha_d));
    for (int j = tid; j < n; j += threads)
      st_dd(d.xh, d.xl, j, dd_add(ld_dd(d.xh, d.xl, j), dd_mul_d(ld_dd(d.dxh, d.dxl, j), alpha)));
    for (int r = tid; r < m; r += threads) {
      d.w[r] += alpha * d.dw[r];
      st_dd(d.zh, d.zl, r, dd_add(ld_dd(d.zh, d.zl, r), dd_mul_d(ld_dd(d.dzh, d.dzl, r), alpha)));
    }
    if (tid == 0 && it < SOV_HISTORY_MAX) d.out->step_hist[it] = alpha;
    cluster.sync();
  }
  cluster.sync();  // no CTA leaves while another may still write its shared memory
}

// Starting point: x = -Q^-1 c (the unconstrained minimiser), slack w = Ax - b shifted into the
// interior (by 1.5 times its most negative entry), z = 1, then both shifted by half the
// complementarity over the other's sum so that the products w_r z_r start balanced (Mehrotra's
// recipe, Mehrotra 1992, section 7).
__global__ void k_xband_start(XbDev d) {
  // one CTA: the shift needs the minimum of w and the sums
  __shared__ double red[4 * 32];
  __shared__ double s_shift, s_dw, s_dz;
  const int tid = threadIdx.x, n = d.n, m = d.m;
  for (int j = tid; j < n; j += blockDim.x) {
    d.xh[j] = -d.c[j] / d.q[j];
    d.xl[j] = 0.0;
  }
  __syncthreads();
  double v[1] = {INFINITY};
  for (int r = tid; r < m; r += blockDim.x) {
    const dd wr = dd_add_d(row_dot(d, r, d.xh, d.xl), -d.b[r]);
    d.w[r] = wr.hi;
    v[0] = fmin(v[0], wr.hi);
  }
  const int opmin[1] = {2};
  block_reduce<1>(v, opmin, red);
  if (tid == 0) s_shift = fmax(-1.5 * v[0], 0.0);
  __syncthreads();
  double s[3] = {0.0, 0.0, 0.0};  // w'z, sum w, sum z
  for (int r = tid; r < m; r += blockDim.x) {
    d.w[r] += s_shift;
    s[0] += d.w[r];
    s[1] += d.w[r];
    s[2] += 1.0;
  }
  const int opsum[3] = {0, 0, 0};
  block_reduce<3>(s, opsum, red);
  if (tid == 0) {
    const bool flat = !(s[0] > 0.0);  // the unconstrained minimiser sits on every row's boundary
    s_dw = flat ? 1.0 : 0.5 * s[0] / s[2];
    s_dz = flat ? 1.0 : 0.5 * s[0] / s[1];
  }
  __syncthreads();
  for (int r = tid; r < m; r += blockDim.x) {
    d.w[r] += s_dw;
    d.zh[r] = 1.0 + s_dz;
    d.zl[r] = 0.0;
  }
}

// One cluster of kXbCluster CTAs (an opt-in size), or of 8 where the device cannot place that one. Up to kXbSmall
// columns 4: its barriers and reductions cost less, and the passes gain nothing from more (4 / 16 CTAs: 3 columns
// 0.138 / 0.179 ms, 20 0.364 / 0.421, 200 1.51 / 1.59, 1000 3.81 / 3.92; 1500 of half-bandwidth 2 1.15 / 1.14).
template <int KD>
void launch_ipm(const XbDev& d, cudaStream_t st) {
  static int ctas[kMaxDevices] = {};
  int dev = 0;
  SOV_CUDA(cudaGetDevice(&dev));
  if (dev >= kMaxDevices) throw std::runtime_error("double-double QP path: device index beyond the supported 64");
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kXbThreads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  once_per_device(reinterpret_cast<const void*>(k_xband_ipm<KD>), [&] {
    SOV_CUDA(cudaFuncSetAttribute(k_xband_ipm<KD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    at.val.clusterDim.x = kXbCluster;
    cfg.gridDim = dim3(kXbCluster);
    int placed = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&placed, k_xband_ipm<KD>, &cfg);
    if (e != cudaSuccess) (void)cudaGetLastError();
    ctas[dev] = e == cudaSuccess && placed > 0 ? kXbCluster : 8;
  });
  {
    std::lock_guard<std::mutex> g(once_mutex());  // the write above happened under this lock
    at.val.clusterDim.x = static_cast<unsigned>(d.n <= kXbSmall ? kXbSmallCluster : ctas[dev]);
  }
  cfg.gridDim = dim3(at.val.clusterDim.x);
  SOV_CUDA(cudaLaunchKernelEx(&cfg, k_xband_ipm<KD>, d));
}

template <class T>
struct XbBuf {
  T* p = nullptr;
  cudaStream_t st = nullptr;
  XbBuf(size_t count, cudaStream_t s) : st(s) {
    SOV_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&p), sizeof(T) * std::max<size_t>(count, 1), st));
  }
  ~XbBuf() {
    if (p) cudaFreeAsync(p, st);
  }
  XbBuf(const XbBuf&) = delete;
  XbBuf& operator=(const XbBuf&) = delete;
  void put(const std::vector<T>& h) {
    if (!h.empty()) SOV_CUDA(cudaMemcpyAsync(p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, st));
  }
};

}  // namespace

bool xband_prepare(const sov_model& p, XBandModel* out) {
  if (const char* off = std::getenv("SOVEREIGN_QP_DISABLE"))
    if ((std::string(",") + off + ",").find(",xband,") != std::string::npos) return false;
  const int n = p.n, m = p.m;
  if (!p.q_col_ptr || p.maximize || n < 1 || m < 1) return false;
  XBandModel& x = *out;
  x = XBandModel{};
  x.n = n;
  x.m = m;
  x.q.assign(n, 0.0);
  for (int j = 0; j < n; ++j)
    for (int k = p.q_col_ptr[j]; k < p.q_col_ptr[j + 1]; ++k) {
      if (p.q_row_idx[k] != j) return false;  // a coupling term
      x.q[j] += p.q_values[k];
    }
  for (int j = 0; j < n; ++j) {
    if (!(x.q[j] > 0.0) || !std::isfinite(x.q[j])) return false;
    if (p.lb && p.lb[j] > -1e29) return false;  // only free variables
    if (p.ub && p.ub[j] < 1e29) return false;
  }
  x.row_sign.resize(m);
  for (int i = 0; i < m; ++i) {
    if (p.sense[i] == SOV_EQ) return false;
    x.row_sign[i] = p.sense[i] == SOV_GE ? 1 : -1;
  }
  // rows: sum duplicates, span check
  std::vector<std::vector<std::pair<int, double>>> rows(m);
  for (int j = 0; j < n; ++j)
    for (int k = p.col_ptr[j]; k < p.col_ptr[j + 1]; ++k) {
      auto& row = rows[p.row_idx[k]];
      const double v = x.row_sign[p.row_idx[k]] * p.values[k];
      if (!row.empty() && row.back().first == j) row.back().second += v;
      else row.push_back({j, v});
    }
  int kd = 0;
  for (int i = 0; i < m; ++i) {
    if (rows[i].empty()) continue;
    kd = std::max(kd, rows[i].back().first - rows[i].front().first);
    if (kd > kXBandMaxKd) return false;
  }
  x.kd = std::max(1, kd);
  x.row_ptr.assign(m + 1, 0);
  for (int i = 0; i < m; ++i) {
    for (const auto& e : rows[i]) {
      x.col_idx.push_back(e.first);
      x.row_val.push_back(e.second);
    }
    x.row_ptr[i + 1] = static_cast<int32_t>(x.col_idx.size());
  }
  x.col_ptr.assign(n + 1, 0);
  for (int i = 0; i < m; ++i)
    for (const auto& e : rows[i]) x.col_ptr[e.first + 1]++;
  for (int j = 0; j < n; ++j) x.col_ptr[j + 1] += x.col_ptr[j];
  x.row_idx.resize(x.col_idx.size());
  x.col_val.resize(x.col_idx.size());
  {
    std::vector<int32_t> at(x.col_ptr.begin(), x.col_ptr.end() - 1);
    for (int i = 0; i < m; ++i)
      for (const auto& e : rows[i]) {
        x.row_idx[at[e.first]] = i;
        x.col_val[at[e.first]++] = e.second;
      }
  }
  x.c.assign(n, 0.0);
  for (int j = 0; j < n; ++j) x.c[j] = p.obj ? p.obj[j] : 0.0;
  x.b.resize(m);
  for (int i = 0; i < m; ++i) x.b[i] = x.row_sign[i] * p.rhs[i];
  x.obj_constant = p.obj_constant;
  return true;
}

int solve_xband(const sov_model& model, const XBandModel& xb, const sov_options& opt, sov_result* r,
                cudaStream_t st, EngineStats* stats) {
  const int n = xb.n, m = xb.m, kd = xb.kd;
  const size_t nnz = xb.col_idx.size();
  XbBuf<int32_t> row_ptr(m + 1, st), col_idx(nnz, st), col_ptr(n + 1, st), row_idx(nnz, st);
  XbBuf<double> row_val(nnz, st), col_val(nnz, st), q(n, st), c(n, st), b(m, st);
  row_ptr.put(xb.row_ptr);
  col_idx.put(xb.col_idx);
  col_ptr.put(xb.col_ptr);
  row_idx.put(xb.row_idx);
  row_val.put(xb.row_val);
  col_val.put(xb.col_val);
  q.put(xb.q);
  c.put(xb.c);
  b.put(xb.b);
  // levels of the odd-even reduction over blocks of kd columns
  XbDev d{};
  d.size[0] = ceil_div(n, kd);
  d.off[0] = 0;
  d.levels = 1;
  while (d.size[d.levels - 1] > 1) {
    d.size[d.levels] = (d.size[d.levels - 1] + 1) / 2;
    d.off[d.levels] = d.off[d.levels - 1] + d.size[d.levels - 1];
    ++d.levels;
  }
  d.slots = d.off[d.levels - 1] + 1;
  if (const char* e = std::getenv("SOVEREIGN_XBAND_SEGMENTS")) d.natural = std::atoi(e) == 1 ? 1 : 0;
  // n-vectors: xh xl rd; dx padded to whole blocks: dxh dxl; m-vectors: zh zl w th rph rpl rcw uh ul dw
  // dzh dzl dwa dza; per block slot: D, L triangles, B X U V W, F Q I
  const size_t nv = 3, mv = 14, np = static_cast<size_t>(d.size[0]) * kd;
  const size_t per_slot = 2 * (static_cast<size_t>(kd) * (kd + 1) / 2 + static_cast<size_t>(kd) * (kd - 1) / 2 +
                               5 * static_cast<size_t>(kd) * kd + 3 * static_cast<size_t>(kd));
  XbBuf<double> work(nv * n + 2 * np + mv * m + per_slot * d.slots, st);
  XbBuf<int> bad(1, st);
  SOV_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(int), st));
  XbBuf<XbOut> out(1, st);
  SOV_CUDA(cudaMemsetAsync(out.p, 0, sizeof(XbOut), st));
  d.n = n;
  d.m = m;
  d.max_iter = std::max(1, opt.max_iterations);
  d.row_ptr = row_ptr.p;
  d.col_idx = col_idx.p;
  d.col_ptr = col_ptr.p;
  d.row_idx = row_idx.p;
  d.row_val = row_val.p;
  d.col_val = col_val.p;
  d.q = q.p;
  d.c = c.p;
  d.b = b.p;
  d.obj_constant = xb.obj_constant;
  double bn = 0.0, cn = 0.0;
  for (double v : xb.b) bn = std::max(bn, std::fabs(v));
  for (double v : xb.c) cn = std::max(cn, std::fabs(v));
  d.bnorm = std::max(1.0, bn);
  d.cnorm = std::max(1.0, cn);  // the slack columns' zero costs do not change max |c|
  d.feas_tol = opt.feasibility_tol;
  d.opt_tol = opt.optimality_tol;
  d.tau = opt.fraction_to_boundary;
  double* wp = work.p;
  auto take = [&wp](size_t count) {
    double* q0 = wp;
    wp += count;
    return q0;
  };
  d.xh = take(n);
  d.xl = take(n);
  d.rd = take(n);
  d.dxh = take(np);
  d.dxl = take(np);
  d.zh = take(m);
  d.zl = take(m);
  d.w = take(m);
  d.th = take(m);
  d.rph = take(m);
  d.rpl = take(m);
  d.rcw = take(m);
  d.uh = take(m);
  d.ul = take(m);
  d.dw = take(m);
  d.dzh = take(m);
  d.dzl = take(m);
  d.dwa = take(m);
  d.dza = take(m);
  const size_t S = static_cast<size_t>(d.slots), tri = static_cast<size_t>(kd) * (kd + 1) / 2, full = static_cast<size_t>(kd) * kd;
  auto pair = [&](double*& h, double*& l, size_t comps) {
    h = take(comps * S);
    l = take(comps * S);
  };
  pair(d.Dh, d.Dl, tri);
  pair(d.Bh, d.Bl, full);
  pair(d.Fh, d.Fl, kd);
  pair(d.Lh, d.Ll, tri - kd);
  pair(d.Ih, d.Il, kd);
  pair(d.Xh, d.Xl, full);
  pair(d.Uh, d.Ul, full);
  pair(d.Vh, d.Vl, full);
  pair(d.Wh, d.Wl, full);
  pair(d.Qh, d.Ql, kd);
  d.bad = bad.p;
  d.out = out.p;
  cudaEvent_t e0, e1;
  SOV_CUDA(cudaEventCreate(&e0));
  SOV_CUDA(cudaEventCreate(&e1));
  SOV_CUDA(cudaEventRecord(e0, st));
  k_xband_start<<<1, 1024, 0, st>>>(d);
  SOV_LAUNCH_CHECK();
  switch (kd) {
    case 1: launch_ipm<1>(d, st); break;
    case 2: launch_ipm<2>(d, st); break;
    case 3: launch_ipm<3>(d, st); break;
    default: launch_ipm<4>(d, st); break;
  }
  SOV_CUDA(cudaEventRecord(e1, st));
  XbOut o;
  std::vector<double> x(n), z(m);
  SOV_CUDA(cudaMemcpyAsync(&o, out.p, sizeof(XbOut), cudaMemcpyDeviceToHost, st));
  SOV_CUDA(cudaMemcpyAsync(x.data(), d.xh, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
  SOV_CUDA(cudaMemcpyAsync(z.data(), d.zh, sizeof(double) * m, cudaMemcpyDeviceToHost, st));
  SOV_CUDA(cudaStreamSynchronize(st));
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (stats) {
    stats->launches += 2;
    stats->factorizations += o.iterations;
    stats->kernel_ms += ms;
  }
  r->status = o.status;
  r->iterations = o.iterations;
  r->has_objective_value = o.status == SOV_OPTIMAL ? 1 : 0;
  r->duality_gap = o.gap;
  r->primal_residual = o.p_res;
  r->dual_residual = o.d_res;
  r->n_ipm = n + m;
  r->m_ipm = m;
  r->solve_seconds = ms * 1e-3;
  double obj = model.obj_constant;
  for (int j = 0; j < n; ++j) obj += xb.c[j] * x[j] + 0.5 * xb.q[j] * x[j] * x[j];
  r->objective_value = obj;
  if (r->primal) std::copy(x.begin(), x.end(), r->primal);
  if (r->dual_col) std::fill(r->dual_col, r->dual_col + n, 0.0);  // free columns carry no bound multiplier
  if (r->dual_row)
    for (int i = 0; i < m; ++i) r->dual_row[i] = xb.row_sign[i] * z[i];
  if (sov_diagnostics* g = r->diagnostics) {
    std::memset(g, 0, sizeof(*g));
    g->structured_qp = 1;
    g->refactorizations = o.iterations;
    g->history_len = o.history_len;
    for (int h = 0; h < o.history_len; ++h) {
      g->history_iterations[h] = o.it_hist[h];
      g->gap_history[h] = o.gap_hist[h];
      g->mu_history[h] = o.mu_hist[h];
      g->objective_history[h] = o.obj_hist[h];
    }
    g->step_history_len = std::min(o.iterations, SOV_HISTORY_MAX);
    for (int h = 0; h < g->step_history_len; ++h) g->primal_step_history[h] = g->dual_step_history[h] = o.step_hist[h];
    g->stall_iteration = -1;
  }
  char desc[200];
  std::snprintf(desc, sizeof desc,
                "x-space Q + A'ZW^-1A, banded LDL^T in double-double on the GPU (order %d, half-bandwidth %d)", n, kd);
  std::string msg;
  if (o.status == SOV_OPTIMAL)
    msg = std::string("Optimal convex QP found by Mehrotra predictor-corrector IPM. KKT system: normal equations, ") +
          desc + ".";
  else if (o.failed)
    msg = std::string("QP-IPM Newton factorization failed (") + desc + ").";
  else
    msg = std::string("QP-IPM iteration limit reached without convergence (") + desc + ").";
  std::snprintf(r->message, sizeof(r->message), "%s", msg.c_str());
  return SOV_OK;
}

}  // namespace sov
