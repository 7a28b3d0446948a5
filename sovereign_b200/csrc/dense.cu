// dense.cu -- dense normal-matrix path on the GPU.
//
// Assembly: one gather pass over a precomputed contribution map (no atomics, deterministic).
// Factorization: blocked right-looking Cholesky, 64-wide panels; one CTA factors a diagonal block
// in shared memory and inverts it, the panel below is L_ik = A_ik L_kk^-T (a GEMM with the
// inverse), and the trailing lower triangle gets A_ij -= L_ik L_jk^T. One launch per panel does
// both as flag-ordered work items, the next diagonal block's factor among them (look-ahead).
// Solves: dataflow triangular solves, one cooperative launch per direction; row block i waits
// (bounded) for the values of the blocks it depends on, so the off-diagonal GEMV work of all
// blocks overlaps and only the 64x64 diagonal products sit on the critical path.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <stdexcept>

#include "common.cuh"
#include "dense.cuh"

namespace sov {

template <class T>
__device__ __forceinline__ T big_pivot();
template <>
__device__ __forceinline__ double big_pivot<double>() {
  return kBigPivotD;
}
template <>
__device__ __forceinline__ float big_pivot<float>() {
  return kBigPivotF;
}

__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }
// four consecutive elements from 16-byte-aligned shared memory
__device__ __forceinline__ void load4(const double* p, double v[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}
__device__ __forceinline__ void load4(const float* p, float v[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = a.z;
  v[3] = a.w;
}
// two consecutive elements, aligned to their size together, widened to double
__device__ __forceinline__ void load2(const double* p, double (&v)[2]) {
  const double2 a = *reinterpret_cast<const double2*>(p);
  v[0] = a.x;
  v[1] = a.y;
}
__device__ __forceinline__ void load2(const float* p, double (&v)[2]) {
  const float2 a = *reinterpret_cast<const float2*>(p);
  v[0] = a.x;
  v[1] = a.y;
}
// sixteen consecutive elements from 16-byte-aligned global memory, widened to double
__device__ __forceinline__ void load16(const double* p, double v[16]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double2 a = reinterpret_cast<const double2*>(p)[k];
    v[2 * k] = a.x;
    v[2 * k + 1] = a.y;
  }
}
__device__ __forceinline__ void load16(const float* p, double v[16]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4 a = reinterpret_cast<const float4*>(p)[k];
    v[4 * k] = a.x;
    v[4 * k + 1] = a.y;
    v[4 * k + 2] = a.z;
    v[4 * k + 3] = a.w;
  }
}

__device__ __forceinline__ double column_weight(int mode, int k, const double* x, const double* s,
                                                const double* qdiag, const uint8_t* free_col) {
  if (mode == kWeightOnes) return 1.0;
  const double xk = fmax(x[k], 1e-16), sk = fmax(s[k], 1e-16);
  if (mode == kWeightLp) return xk / sk;
  if (mode == kWeightTheta) return sk / xk;
  const double h = free_col[k] ? 0.0 : sk / xk;
  return 1.0 / (qdiag[k] + h);
}

// layout_ld > 0: dense column-major with that leading dimension; layout_ld < 0: band storage
// with -layout_ld = m (diagonal offset major).
template <class T>
__global__ void k_assemble(AssemblyDev am, const double* __restrict__ x, const double* __restrict__ s,
                           const double* __restrict__ qdiag, const uint8_t* __restrict__ free_col, int mode,
                           double reg, T* __restrict__ out, double* __restrict__ diag_out, int m, int layout_ld) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= am.ntargets) return;
  double acc = 0.0;
  for (int p = am.ptr[t]; p < am.ptr[t + 1]; ++p)
    acc += am.w[p] * column_weight(mode, am.col[p], x, s, qdiag, free_col);
  const int64_t tg = am.target[t];
  int row = -1;
  if (layout_ld > 0) {
    const int r = static_cast<int>(tg % layout_ld), c = static_cast<int>(tg / layout_ld);
    if (r == c) row = r;
  } else if (tg < m) {
    row = static_cast<int>(tg);
  }
  if (row >= 0) {
    acc += reg;
    diag_out[row] = acc;
  }
  out[tg] = static_cast<T>(acc);
}

template <class T>
void launch_assemble(const AssemblyDev& am, const double* x, const double* s, const double* qdiag,
                     const uint8_t* free_col, int mode, double reg, T* out, double* diag_out, int m,
                     int layout_ld, cudaStream_t st) {
  if (am.ntargets == 0) return;
  k_assemble<T><<<ceil_div(am.ntargets, 256), 256, 0, st>>>(am, x, s, qdiag, free_col, mode, reg, out, diag_out, m,
                                                           layout_ld);
  SOV_LAUNCH_CHECK();
}

template <class T>
__global__ void k_pad_identity(T* M, int m, int mp) {
  const int i = m + blockIdx.x * blockDim.x + threadIdx.x;
  if (i < mp) M[static_cast<int64_t>(i) * mp + i] = T(1);
}

template <class T>
void launch_dense_clear(T* M, int m, int mp, cudaStream_t st) {
  SOV_CUDA(cudaMemsetAsync(M, 0, sizeof(T) * static_cast<size_t>(mp) * mp, st));
  if (mp > m) {
    k_pad_identity<T><<<ceil_div(mp - m, 128), 128, 0, st>>>(M, m, mp);
    SOV_LAUNCH_CHECK();
  }
}

// ---------------------------------------------------------------------------------------------
// Diagonal block (64 x 64) on 256 threads, right-looking over 8-column panels with look-ahead (one
// barrier per panel), then the blocked inverse of the 64 x 64 factor. Pivots come from one
// reciprocal square root (l_jj = p * rsqrt(p)), whose reciprocal is kept for the panel solves and
// the inverse.
// ---------------------------------------------------------------------------------------------
constexpr int kPanel = 8;
// diagonal factor's shared memory: A and I (64 x 65 each) and two transposed panels (8 x 64 each)
template <class T>
constexpr size_t potrf_smem_bytes() {
  return sizeof(T) * (2 * kNB * (kNB + 1) + 2 * kPanel * kNB);
}

template <int kId, int kCount>
__device__ __forceinline__ void bar_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(kId), "n"(kCount) : "memory");
}

// Row block p (rows 8p..8p+7) of X = L^-1, into I, once L's rows 8p..8p+7 are final in A and the
// earlier row blocks of X are in I, in three steps:
//   x1  X_pp = L_pp^-1, one column per thread (eight threads), by forward substitution;
//   x2  T_pj = sum_{k=j}^{8p-1} L[8p+q][k] X[k][j] for every column j < 8p, one entry at a time
//       from a shared counter, so threads join as they come free; T goes to X's place;
//   x3  X_pj = -X_pp T_pj, one entry per thread, written after a barrier (in place of T).
template <class T>
__device__ __forceinline__ void inverse_x1(const T (*A)[kNB + 1], T (*I)[kNB + 1], const T* rinv, int p, int c) {
  // L_pp x = e_c, right-looking with every index static (x starts as e_c, so the entries above c
  // stay zero)
  const int R = p * kPanel;
  T l[kPanel * (kPanel - 1) / 2], ri[kPanel], x[kPanel];
#pragma unroll
  for (int r = 0; r < kPanel; ++r) {
    ri[r] = rinv[R + r];
    x[r] = r == c ? T(1) : T(0);
#pragma unroll
    for (int k = 0; k < r; ++k) l[r * (r - 1) / 2 + k] = A[R + r][R + k];
  }
#pragma unroll
  for (int k = 0; k < kPanel; ++k) {
    x[k] *= ri[k];
#pragma unroll
    for (int r = k + 1; r < kPanel; ++r) x[r] -= l[r * (r - 1) / 2 + k] * x[k];
  }
#pragma unroll
  for (int r = 0; r < kPanel; ++r) I[R + r][R + c] = x[r];
}

template <class T>
__device__ __forceinline__ void inverse_x2(const T (*A)[kNB + 1], T (*I)[kNB + 1], int p, int* next) {
  const int R = p * kPanel;
  for (int e = atomicAdd(next, 1); e < kPanel * R; e = atomicAdd(next, 1)) {
    const int q = e % kPanel, j = e / kPanel;
    // by 8-row blocks of X from j's own (X is lower triangular: rows above j in it are zero),
    // each block's 16 loads issued together
    T a0 = T(0), a1 = T(0);
    for (int k0 = j & ~(kPanel - 1); k0 < R; k0 += kPanel) {
      T l[kPanel], x[kPanel];
#pragma unroll
      for (int t = 0; t < kPanel; ++t) {
        l[t] = A[R + q][k0 + t];
        x[t] = I[k0 + t][j];
      }
#pragma unroll
      for (int t = 0; t < kPanel; t += 2) {
        a0 += l[t] * x[t];
        a1 += l[t + 1] * x[t + 1];
      }
    }
    I[R + q][j] = a0 + a1;
  }
}

// kThreads threads from u = 0, on barrier kBar; every 8p * 8 <= 2 * kThreads
template <int kThreads, int kBar, class T>
__device__ __forceinline__ void inverse_x3(T (*I)[kNB + 1], int p, int u) {
  const int R = p * kPanel;
  T x[2];
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const int e = u + v * kThreads;
    if (e < kPanel * R) {
      const int q = e % kPanel, j = e / kPanel;
      T acc = T(0);
#pragma unroll
      for (int r = 0; r < kPanel; ++r)
        if (r <= q) acc += I[R + q][R + r] * I[R + r][j];
      x[v] = -acc;
    }
  }
  bar_sync<kBar, kThreads>();
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const int e = u + v * kThreads;
    if (e < kPanel * R) I[R + e % kPanel][e / kPanel] = x[v];
  }
}

// One 8-column panel of the diagonal block on the 64 threads of warps 0-1: every one of them
// factors the 8 x 8 diagonal block (rows/cols k0..k0+7 of A) in registers with the same
// arithmetic (no exchange on the pivot chain, the pivot rule without branches); then (after
// barrier 2, where warps 2-7 signal that the rows below are updated, if kWaitRows) the thread
// with a row below (row k0 + 8 + tid) solves it against that factor and stores it to A and,
// transposed, to Lw (Lw[c][i] = L[i][k0 + c]). Warps 0 and 1 store halves of the factored 8 x 8
// block and the pivot reciprocals.
template <bool kWaitRows, class T>
__device__ __forceinline__ void factor_panel(T (*A)[kNB + 1], T (*Lw)[kNB], T* rinv, const double* dref, int k0,
                                             int r0, int m, double drop_tol, int& drops, int& bad) {
  const int tid = threadIdx.x;
  const bool has_row = tid < kNB - k0 - kPanel;
  T d[kPanel][kPanel], dinv[kPanel];
  double thr[kPanel];
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    thr[j] = drop_tol * dref[k0 + j];
#pragma unroll
    for (int c = 0; c <= j; ++c) d[j][c] = A[k0 + j][k0 + c];
  }
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    const T p = d[j][j];
    const double pd = static_cast<double>(p);
    // dependent row (sparse_ldlt.cpp:165-173): pivot not finite, or at most tol * |diag|
    const bool finite = fabs(pd) <= DBL_MAX;
    const bool drop = !(finite && pd > thr[j]);
    bad |= !finite;
    drops += (drop && r0 + k0 + j < m);
    const T inv_p = rsqrt_t(p);
    const T inv = drop ? T(1) / big_pivot<T>() : inv_p;
    d[j][j] = drop ? big_pivot<T>() : p * inv_p;
    dinv[j] = inv;
#pragma unroll
    for (int q = j + 1; q < kPanel; ++q) d[q][j] *= inv;
#pragma unroll
    for (int q = j + 1; q < kPanel; ++q)
#pragma unroll
      for (int k = j + 1; k <= q; ++k) d[q][k] -= d[q][j] * d[k][j];
  }
  if (kWaitRows) asm volatile("bar.sync 2, 256;" ::: "memory");
  if (has_row) {
    const int i = k0 + kPanel + tid;
    T r[kPanel];
#pragma unroll
    for (int c = 0; c < kPanel; ++c) r[c] = A[i][k0 + c];
#pragma unroll
    for (int c = 0; c < kPanel; ++c) {
      r[c] *= dinv[c];
#pragma unroll
      for (int e = c + 1; e < kPanel; ++e) r[e] -= r[c] * d[e][c];
    }
#pragma unroll
    for (int c = 0; c < kPanel; ++c) {
      A[i][k0 + c] = r[c];
      Lw[c][i] = r[c];
    }
  }
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < kPanel / 2; ++q) {
      rinv[k0 + q] = dinv[q];
#pragma unroll
      for (int c = 0; c <= q; ++c) A[k0 + q][k0 + c] = d[q][c];
    }
  } else if (tid == 32) {
#pragma unroll
    for (int q = kPanel / 2; q < kPanel; ++q) {
      rinv[k0 + q] = dinv[q];
#pragma unroll
      for (int c = 0; c <= q; ++c) A[k0 + q][k0 + c] = d[q][c];
    }
  }
}

// The diagonal block's lower triangle from M into A (upper entries zero); 256 threads.
template <class T>
__device__ __forceinline__ void potrf_load(const T* __restrict__ M, int ld, int kb, unsigned char* potrf_raw) {
  T(*A)[kNB + 1] = reinterpret_cast<T(*)[kNB + 1]>(potrf_raw);
  const int tid = threadIdx.x, r0 = kb * kNB;
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // 8 loads in flight per thread
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = tid + 256 * (8 * h + u), c = idx / kNB, r = idx % kNB;
      v[u] = r >= c ? M[static_cast<int64_t>(r0 + c) * ld + r0 + r] : T(0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = tid + 256 * (8 * h + u);
      A[idx % kNB][idx / kNB] = v[u];
    }
  }
}

// Factor and invert the diagonal block held in A (the first 64 x 65 elements of `potrf_raw`,
// lower triangle, upper entries zero); stores L to M and L^-1 to Linv. Runs on a CTA of 256
// threads; `potrf_raw` is potrf_smem_bytes<T>() of dynamic shared memory.
// Panels with look-ahead: while warps 0-1 apply panel p's update to panel p+1's diagonal block and
// factor it, warps 2-7 apply panel p's update to the rows below it (handed over on a barrier the
// row solves wait on) and then to the trailing triangle right of panel p+1, so each panel costs
// one block-wide barrier and the longer of the two chains. Warps 2-7 then also compute row block p
// of the inverse (rows of L up to panel p are final), so only the last row block follows the
// panels.
template <class T>
__device__ void potrf_core(T* __restrict__ M, int ld, int kb, const double* __restrict__ diag, int m,
                           T* __restrict__ Linv, int* drop_count, int* fail, double drop_tol,
                           unsigned char* potrf_raw) {
  T(*A)[kNB + 1] = reinterpret_cast<T(*)[kNB + 1]>(potrf_raw);
  T(*I)[kNB + 1] = reinterpret_cast<T(*)[kNB + 1]>(potrf_raw + sizeof(T) * kNB * (kNB + 1));
  __shared__ T rinv[kNB];
  __shared__ double dref[kNB];
  __shared__ int x2_next[kNB / kPanel];  // per row block of the inverse: next entry of its x2 step
  const int tid = threadIdx.x;
  const int r0 = kb * kNB;
  if (tid < kNB) dref[tid] = r0 + tid < m ? fabs(diag[r0 + tid]) : 1.0;
  if (tid < kNB / kPanel) x2_next[tid] = 0;
  __syncthreads();
  int drops = 0, bad = 0;
  // two panels' columns below their diagonal blocks, transposed (Lt[c][i] = L[i][k0 + c]), so an
  // update reads consecutive rows per vector load
  T(*Lt0)[kNB] = reinterpret_cast<T(*)[kNB]>(potrf_raw + 2 * sizeof(T) * kNB * (kNB + 1));
  T(*Lt1)[kNB] = Lt0 + kPanel;
  // warps 2-7: 4 x 4 tile (ti, tj) of the trailing update, u = ti (ti + 1) / 2 + tj, the same for
  // every panel (a triangle of nt tile rows uses u below nt (nt + 1) / 2)
  const int u = tid - kNB;
  int ti = 0, tj = 0;
  if (u >= 0) {
    ti = static_cast<int>((sqrtf(8.0f * u + 1.0f) - 1.0f) * 0.5f);
    while (ti * (ti + 1) / 2 > u) --ti;
    while ((ti + 1) * (ti + 2) / 2 <= u) ++ti;
    tj = u - ti * (ti + 1) / 2;
  }
  int dq = 0;  // tid < 36: entry (dq, dc) of an 8 x 8 lower triangle
  while (tid < kPanel * (kPanel + 1) / 2 && (dq + 1) * (dq + 2) / 2 <= tid) ++dq;
  const int dc = tid - dq * (dq + 1) / 2;
  if (tid < kNB) factor_panel<false, T>(A, Lt0, rinv, dref, 0, r0, m, drop_tol, drops, bad);
  __syncthreads();
  for (int p = 0; p + 1 < kNB / kPanel; ++p) {
    const int K0 = (p + 1) * kPanel, K1 = K0 + kPanel;  // panel p+1's first column, and the next
    T(*Lc)[kNB] = (p & 1) ? Lt1 : Lt0;                 // panel p
    T(*Ln)[kNB] = (p & 1) ? Lt0 : Lt1;                 // panel p + 1
    if (tid < kNB) {
      // panel p's update of panel p+1's diagonal block, one entry per thread, shared through A
      if (tid < kPanel * (kPanel + 1) / 2) {
        T a = A[K0 + dq][K0 + dc];
#pragma unroll
        for (int k = 0; k < kPanel; ++k) a -= Lc[k][K0 + dq] * Lc[k][K0 + dc];
        A[K0 + dq][K0 + dc] = a;
      }
      asm volatile("bar.sync 1, 64;" ::: "memory");  // warps 0-1: the diagonal block is updated
      factor_panel<true, T>(A, Ln, rinv, dref, K0, r0, m, drop_tol, drops, bad);
    } else {
      // panel p's update of panel p+1's columns below its diagonal block (two entries per
      // thread), signalled to warps 0-1 on barrier 2 without waiting
      {
        const int i = K1 + (u >> 2), c0 = (u & 3) * 2;
        if (i < kNB) {
          T li[kPanel];
#pragma unroll
          for (int k = 0; k < kPanel; ++k) li[k] = Lc[k][i];
#pragma unroll
          for (int c = c0; c < c0 + 2; ++c) {
            T a = A[i][K0 + c];
#pragma unroll
            for (int k = 0; k < kPanel; ++k) a -= li[k] * Lc[k][K0 + c];
            A[i][K0 + c] = a;
          }
        }
      }
      asm volatile("bar.arrive 2, 256;" ::: "memory");
      // row block p of the inverse: x1 on threads that have no tiles, x2 shared by all
      if (u >= 88 && u < 88 + kPanel) inverse_x1<T>(A, I, rinv, p, u - 88);
      // panel p's update of the trailing triangle (rows and columns from K1)
      const int nt = (kNB - K1) / 4;
      if (ti < nt) {
        const int i0 = K1 + 4 * ti, j0 = K1 + 4 * tj;
        T acc[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[q][v] = A[i0 + q][j0 + v];
#pragma unroll
        for (int k = 0; k < kPanel; ++k) {
          T li[4], lj[4];
          load4(&Lc[k][i0], li);
          load4(&Lc[k][j0], lj);
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[q][v] -= li[q] * lj[v];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int v = 0; v < 4; ++v)
            if (j0 + v <= i0 + q) A[i0 + q][j0 + v] = acc[q][v];
      }
      inverse_x2<T>(A, I, p, &x2_next[p]);
      if (p > 0) {
        bar_sync<3, 192>();
        inverse_x3<192, 3, T>(I, p, u);
      }
    }
    __syncthreads();
  }
  // the inverse's last row block, on all threads
  constexpr int kLast = kNB / kPanel - 1;
  if (tid >= 256 - kPanel) inverse_x1<T>(A, I, rinv, kLast, tid - (256 - kPanel));
  inverse_x2<T>(A, I, kLast, &x2_next[kLast]);
  __syncthreads();
  inverse_x3<256, 0, T>(I, kLast, tid);
  __syncthreads();
#pragma unroll 8
  for (int v = 0; v < kNB * kNB / 256; ++v) {
    const int idx = tid + 256 * v, cc = idx / kNB, r = idx % kNB;
    if (r >= cc) M[static_cast<int64_t>(r0 + cc) * ld + r0 + r] = A[r][cc];
    Linv[static_cast<int64_t>(kb) * kNB * kNB + idx] = r >= cc ? I[r][cc] : T(0);
  }
  if (tid == 0) {
    if (drops) atomicAdd(drop_count, drops);
    if (bad) atomicExch(fail, 1);
  }
}

template <class T>
__device__ __forceinline__ void potrf_block(T* __restrict__ M, int ld, int kb, const double* __restrict__ diag, int m,
                                            T* __restrict__ Linv, int* drop_count, int* fail, double drop_tol,
                                            unsigned char* potrf_raw) {
  potrf_load<T>(M, ld, kb, potrf_raw);
  potrf_core<T>(M, ld, kb, diag, m, Linv, drop_count, fail, drop_tol, potrf_raw);
}

template <class T>
__global__ void __launch_bounds__(256) k_potrf_diag(T* __restrict__ M, int ld, int kb, const double* __restrict__ diag,
                                                    int m, T* __restrict__ Linv, int* drop_count, int* fail,
                                                    double drop_tol, unsigned* tickets) {
  extern __shared__ __align__(16) unsigned char potrf_raw[];
  if (tickets != nullptr && threadIdx.x == 0) *tickets = 0u;
  potrf_block<T>(M, ld, kb, diag, m, Linv, drop_count, fail, drop_tol, potrf_raw);
}

// Rows of the slices in shared memory: 68 doubles apart, so that an MMA fragment's 8 x 4 entries (four
// rows, eight entries each) meet in no bank more than twice.
constexpr int kSliceLd = 68;

// acc[p][q] += sum_k Xs[k][tx + 16 p] Ys[k][ty + 16 q], tx = tid % 16, ty = tid / 16 (256 threads):
// a half-warp reads 16 consecutive entries of Xs (one wavefront) and one entry of Ys (broadcast),
// and its results are 16 consecutive rows of a column-major tile (coalesced stores)
template <class T>
__device__ __forceinline__ void tile_nt(const T (*Xs)[kSliceLd], const T (*Ys)[kSliceLd], T (&acc)[4][4]) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 8
  for (int k = 0; k < kNB; ++k) {
    T a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = Xs[k][tx + 16 * q];
      b[q] = Ys[k][ty + 16 * q];
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] += a[p] * b[q];
  }
}

// Two 64 x 64 slices into shared memory, dst[k][r] = src[k * ld + r], on 256 threads with 16
// loads in flight per thread; kBypassL1 reads past L1 (data written by other CTAs of this launch).
template <bool kBypassL1, class T>
__device__ __forceinline__ void load_slices(T (*Xs)[kSliceLd], const T* __restrict__ xsrc, int64_t xld, T (*Ys)[kSliceLd],
                                            const T* __restrict__ ysrc, int64_t yld) {
  const int tid = threadIdx.x;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    T vx[8], vy[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = tid + 256 * (8 * h + u), k = idx / kNB, r = idx % kNB;
      vx[u] = kBypassL1 ? __ldcg(xsrc + k * xld + r) : xsrc[k * xld + r];
      vy[u] = kBypassL1 ? __ldcg(ysrc + k * yld + r) : ysrc[k * yld + r];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int idx = tid + 256 * (8 * h + u);
      Xs[idx / kNB][idx % kNB] = vx[u];
      Ys[idx / kNB][idx % kNB] = vy[u];
    }
  }
}

// Products of 64 x 64 slices where a triangle of them is zero or not wanted, in 8 x 8 FP64 MMA tiles: 36 of
// the 64 tiles' work, which is what bounds them (one SM: 4096 cycles for the whole product). Warp w has
// row block rb; its lane (q, t) = (lane / 4, lane % 4) holds entries (8 rb + q, 8 cb + 2t) and the next one
// of column block cb in c[cb].
__device__ __forceinline__ void mma_step(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
// c += X Y' with Y lower triangular: Xs[k][r], Ys[k][col] = 0 for k > col
__device__ __forceinline__ void product_lower_factor(const double (*Xs)[kSliceLd], const double (*Ys)[kSliceLd], int rb,
                                                     double (&c)[8][2]) {
  const int q = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  double a[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) a[k] = Xs[4 * k + t][8 * rb + q];
#pragma unroll
  for (int k = 0; k < 16; ++k)
#pragma unroll
    for (int cb = k / 2; cb < 8; ++cb) mma_step(c[cb], a[k], Ys[4 * k + t][8 * cb + q]);
}
// the column blocks cb <= rb of c += X X'
__device__ __forceinline__ void product_lower_result(const double (*Xs)[kSliceLd], int rb, double (&c)[8][2]) {
  const int q = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll 4
  for (int k = 0; k < 16; ++k) {
    const double a = Xs[4 * k + t][8 * rb + q];
#pragma unroll
    for (int cb = 0; cb < 8; ++cb)
      if (cb <= rb) mma_step(c[cb], a, Xs[4 * k + t][8 * cb + q]);
  }
}

constexpr long long kSpinLimit = 1ll << 22;  // bounded wait (x >= 64 ns per poll -> > 0.25 s)

__device__ __forceinline__ bool wait_flag(const unsigned* flag, unsigned epoch) {
  long long n = 0;
  while (ld_acquire(flag) != epoch) {
    if (++n > kSpinLimit) return false;
    __nanosleep(64);
  }
  return true;
}

__device__ __forceinline__ void tile_triangle(int t, int& ii, int& jj) {
  // t -> (ii, jj) with 0 <= jj <= ii, t = ii (ii + 1) / 2 + jj
  ii = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((ii + 1) * (ii + 2) / 2 <= t) ++ii;
  while (ii * (ii + 1) / 2 > t) --ii;
  jj = t - ii * (ii + 1) / 2;
}

// One launch per panel kb < nb - 1: the panel solves L_ik = A_ik Linv_kk^T of the R = nb - kb - 1
// row blocks below it and the trailing updates A_ij -= L_ik L_jk^T of the tiles kb < j <= i, as
// R + R (R + 1) / 2 - 1 work items taken in ticket order (an atomic counter):
//   item 0      the look-ahead chain: row block kb + 1's panel solve, then its diagonal tile's
//               update from the solved block still in shared memory, then the factor and inverse
//               of that diagonal block (potrf_block), so the next panel's diagonal factor starts
//               as soon as its own inputs exist rather than after the whole panel;
//   1 .. R-1    the other panel solves, each publishing its row block with a release flag;
//   R ..        the other trailing tiles, each waiting (acquire, bounded) for its two row blocks.
// A trailing tile only waits for panel solves, which never wait and hold lower tickets, so every
// item it waits for was taken by a CTA that is already running. Blocks solved by other CTAs of
// the launch are read past L1 (ld.global.cg).
// Item 0 bounds a launch (the other items finish under it): 43000 cycles at 64 x 64, of which the factor and
// inverse 25000. Its two products take 36 of 64 tiles, the diagonal tile is on its way from the start,
// and the solved block is released only once the factor can begin (its readers have that long).
// Measured per panel at order 2000: 28.6 us before, 24.3 in this form (sums in the same order, same bits).
__global__ void __launch_bounds__(256) k_panel_update(double* __restrict__ M, int ld, int kb, int nb,
                                                      const double* __restrict__ diag, int m, double* __restrict__ Linv,
                                                      int* drop_count, int* fail, double drop_tol, unsigned* flags,
                                                      unsigned stamp, unsigned* tickets, unsigned base) {
  using T = double;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T(*Xs)[kSliceLd] = reinterpret_cast<T(*)[kSliceLd]>(smem_raw);
  T(*Ys)[kSliceLd] = reinterpret_cast<T(*)[kSliceLd]>(smem_raw + sizeof(T) * kNB * kSliceLd);
  __shared__ unsigned item_s;
  __shared__ int ok_s;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  if (tid == 0) item_s = atomicAdd(tickets, 1u) - base;
  __syncthreads();
  const int item = static_cast<int>(item_s);
  const int R = nb - kb - 1, k0 = kb * kNB;
  if (item < R) {
    const int i = kb + 1 + item, r0 = i * kNB;
    const int warp = tid >> 5, q = (tid & 31) >> 2, t = tid & 3;
    // row blocks so dealt that the two warps of a scheduler share 9 tiles of a lower triangle
    const int rb = warp < 4 ? warp : 11 - warp;
    double cur[8][2];  // item 0: the diagonal tile's lower triangle
#pragma unroll
    for (int cb = 0; cb < 8; ++cb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 8 * rb + q, c = 8 * cb + 2 * t + e;
        cur[cb][e] = item == 0 && r >= c ? M[static_cast<int64_t>(r0 + c) * ld + r0 + r] : T(0);
      }
    // Ys[k][c] = Linv[c][k] = Lk[k * 64 + c]
    load_slices<false>(Xs, M + static_cast<int64_t>(k0) * ld + r0, ld, Ys, Linv + static_cast<int64_t>(kb) * kNB * kNB,
                       kNB);
    __syncthreads();
    double acc[8][2] = {};
    product_lower_factor(Xs, Ys, rb, acc);
#pragma unroll
    for (int cb = 0; cb < 8; ++cb)
#pragma unroll
      for (int e = 0; e < 2; ++e) M[static_cast<int64_t>(k0 + 8 * cb + 2 * t + e) * ld + r0 + 8 * rb + q] = acc[cb][e];
    __syncthreads();
    if (item != 0) {
      if (tid == 0) {
        __threadfence();
        st_release(flags + i, stamp);
      }
      return;
    }
    // look-ahead: A_ii - L_ik L_ik^T from the block just solved, straight into the diagonal
    // factor's shared-memory tile, then its factor and inverse
#pragma unroll
    for (int cb = 0; cb < 8; ++cb)
#pragma unroll
      for (int e = 0; e < 2; ++e) Xs[8 * cb + 2 * t + e][8 * rb + q] = acc[cb][e];
    __syncthreads();
    double upd[8][2] = {};
    product_lower_result(Xs, rb, upd);
    __syncthreads();  // Xs, which the factor's tile overlays, is fully read
    T(*A)[kNB + 1] = reinterpret_cast<T(*)[kNB + 1]>(smem_raw);
#pragma unroll
    for (int cb = 0; cb < 8; ++cb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = 8 * rb + q, c = 8 * cb + 2 * t + e;
        A[r][c] = r >= c ? cur[cb][e] - upd[cb][e] : T(0);
      }
    if (tid == 255) {  // every thread's rows were stored before the last barriers
      __threadfence();
      st_release(flags + i, stamp);
    }
    potrf_core<T>(M, ld, kb + 1, diag, m, Linv, drop_count, fail, drop_tol, smem_raw);
    return;
  }
  int ii, jj;
  tile_triangle(item - R + 1, ii, jj);
  const int i = kb + 1 + ii, j = kb + 1 + jj;
  if (tid == 0) ok_s = wait_flag(flags + i, stamp) && wait_flag(flags + j, stamp);
  __syncthreads();
  if (!ok_s) {
    if (tid == 0) atomicExch(fail, 1);
    return;
  }
  const int r0 = i * kNB, c0 = j * kNB;
  load_slices<true>(Xs, M + static_cast<int64_t>(k0) * ld + r0, ld, Ys, M + static_cast<int64_t>(k0) * ld + c0, ld);
  __syncthreads();
  T acc[4][4] = {};
  tile_nt<T>(Xs, Ys, acc);
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int p = 0; p < 4; ++p) M[static_cast<int64_t>(c0 + ty + 16 * q) * ld + r0 + tx + 16 * p] -= acc[p][q];
}

template <class T>
void dense_potrf_block(const DenseSystem<T>& s, int kb, cudaStream_t st) {
  const size_t smem_potrf = potrf_smem_bytes<T>();
  once_per_device((const void*)k_potrf_diag<T>, [&] {
    SOV_CUDA(cudaFuncSetAttribute(k_potrf_diag<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_potrf));
  });
  k_potrf_diag<T><<<1, 256, smem_potrf, st>>>(s.M, s.mp, kb, s.diag, s.m, s.Linv, s.drop_count, s.fail, s.drop_tol,
                                              nullptr);
}

// panel stamps: top bit set (never the zero the flags start from), a generation per
// factorization and the panel index below it
constexpr int kStampPanelBits = 11;
std::atomic<unsigned> g_factor_generation{0};

template <class T>
void dense_cholesky(const DenseSystem<T>& s, cudaStream_t st, int* launches) {
  static_assert(sizeof(T) == sizeof(double), "FP32 factors go through dense_cholesky_tc");
  static_assert(2 * kNB * kSliceLd * sizeof(T) <= potrf_smem_bytes<T>(), "slices larger than the factor's shared memory");
  const size_t smem_potrf = potrf_smem_bytes<T>();
  once_per_device((const void*)k_panel_update, [&] {
    SOV_CUDA(cudaFuncSetAttribute(k_potrf_diag<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_potrf));
    SOV_CUDA(cudaFuncSetAttribute(k_panel_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_potrf));
  });
  if (s.nb >= (1 << kStampPanelBits)) throw std::runtime_error("dense factor: too many row blocks");
  const unsigned gen = (g_factor_generation.fetch_add(1) & ((1u << (31 - kStampPanelBits)) - 1)) << kStampPanelBits;
  // panel 0's diagonal block alone (it also resets the ticket counter); every later one is
  // factored by item 0 of the previous panel's launch
  k_potrf_diag<T><<<1, 256, smem_potrf, st>>>(s.M, s.mp, 0, s.diag, s.m, s.Linv, s.drop_count, s.fail, s.drop_tol,
                                              s.tickets);
  int n = 1;
  unsigned base = 0;
  for (int kb = 0; kb + 1 < s.nb; ++kb) {
    const int R = s.nb - kb - 1;
    const int items = R + R * (R + 1) / 2 - 1;
    const unsigned stamp = 0x80000000u | gen | static_cast<unsigned>(kb);
    k_panel_update<<<items, 256, smem_potrf, st>>>(s.M, s.mp, kb, s.nb, s.diag, s.m, s.Linv, s.drop_count, s.fail,
                                                       s.drop_tol, s.flags, stamp, s.tickets, base);
    base += static_cast<unsigned>(items);
    ++n;
  }
  SOV_LAUNCH_CHECK();
  if (launches) *launches += n;
}

// ---------------------------------------------------------------------------------------------
// Dataflow triangular solves
// ---------------------------------------------------------------------------------------------
// A solved block is handed over by its values alone: the buffer they are published in holds kUnset (a NaN
// no arithmetic produces; a result with those bits is published as the standard NaN) until then, and a
// consumer polls the value it needs. Flags cost a chain step two more trips to L2 (fence and flag on
// one side, flag and then value on the other). A block takes its dependencies one by one, the next tile on
// its way while it waits: taken up to eight to a barrier, the block that publishes next was still busy
// with its run when its last value came. Forward / backward, us a solve:
//                         flags        values, runs of 8    values, one by one
//   FP64, order 2000      71 / 79      56 / 63              31.5 / 39
//   FP32, order 700       27.2 / 25.8  20 / 20              14.3 / 15.7
// Above 148 blocks a CTA takes several rows; 148 rather than 296 CTAs (one per SM, for the registers).
constexpr unsigned long long kUnset = ~0ull;  // cudaMemset 0xFF

__device__ __forceinline__ void publish_value(double* p, double v) {
  unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  if (u == kUnset) u = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}

// bounded (kSpinLimit polls); a wait that gives up sets *err and takes the NaN
__device__ __forceinline__ double wait_value(const double* p, int* err) {
  unsigned long long u = kUnset;
  for (long long n = 0; n < kSpinLimit; ++n) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
    if (u != kUnset) break;
    if (n >= 256) __nanosleep(64);
  }
  if (u == kUnset) atomicExch(err, 1);
  return __longlong_as_double(static_cast<long long>(u));
}

// Forward: L y = r, row block order. z holds r; y goes to Y. X (of the last backward solve) is unset again.
template <class T>
__global__ void __launch_bounds__(256, 1) k_trsv_fwd(const T* __restrict__ M, int ld, const T* __restrict__ Linv, int nb,
                                                  const double* z, double* Y, double* X, int* err) {
  __shared__ double part[4][kNB];
  __shared__ double ys[2][kNB];  // by turns: a block's values are read while the next one's are awaited
  __shared__ double rhs[kNB];
  const int t = threadIdx.x, r = t & (kNB - 1), g = t >> 6;
  for (int i = blockIdx.x; i < nb; i += gridDim.x) {
    // this thread's 16 entries of Linv_ii and of L_{i,i-1} (the last dependency), loaded before any
    // wait: once block i-1 is published, the remaining path has no global loads of L
    double li[16], lp[16];
    const T* Li = Linv + static_cast<int64_t>(i) * kNB * kNB;
#pragma unroll
    for (int u = 0; u < 16; ++u) li[u] = static_cast<double>(Li[(g * 16 + u) * kNB + r]);
    if (i > 0) {
      const T* Lp = M + static_cast<int64_t>((i - 1) * kNB) * ld + i * kNB + r;
#pragma unroll
      for (int u = 0; u < 16; ++u) lp[u] = static_cast<double>(Lp[static_cast<int64_t>(g * 16 + u) * ld]);
    }
    const double zi = t < kNB ? z[i * kNB + t] : 0.0;
    if (t < kNB) X[i * kNB + t] = __longlong_as_double(static_cast<long long>(kUnset));
    double acc = 0.0;
    const T* Lij = M + static_cast<int64_t>(g * 16) * ld + i * kNB + r;
    double next[16];
    if (i > 1) {
#pragma unroll
      for (int u = 0; u < 16; ++u) next[u] = static_cast<double>(Lij[static_cast<int64_t>(u) * ld]);
    }
    for (int j = 0; j + 1 < i; ++j) {  // blocks 0 .. i-2
      double l[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) l[u] = next[u];
      if (j + 2 < i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) next[u] = static_cast<double>(Lij[static_cast<int64_t>((j + 1) * kNB + u) * ld]);
      }
      if (t < kNB) ys[j & 1][t] = wait_value(Y + j * kNB + t, err);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 16; ++u) acc += l[u] * ys[j & 1][g * 16 + u];
    }
    if (i > 0) {
      double(&yl)[kNB] = ys[(i - 1) & 1];
      if (t < kNB) yl[t] = wait_value(Y + (i - 1) * kNB + t, err);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 16; ++u) acc += lp[u] * yl[g * 16 + u];
    }
    part[g][r] = acc;
    __syncthreads();
    if (t < kNB) rhs[t] = zi - (part[0][t] + part[1][t] + part[2][t] + part[3][t]);
    __syncthreads();
    double y = 0.0;
#pragma unroll
    for (int u = 0; u < 16; ++u) y += li[u] * rhs[g * 16 + u];
    part[g][r] = y;
    __syncthreads();
    if (t < kNB) publish_value(Y + i * kNB + t, part[0][t] + part[1][t] + part[2][t] + part[3][t]);
    __syncthreads();  // part and ys are reused by this CTA's next block
  }
}

// Backward: L^T x = y, reverse row block order; x goes to X and z, and Y is unset again.
// Warp w has columns 8w .. 8w+7 of a block, its lane (c, g) rows 16g .. 16g+15 of one of them. The tiles
// before the last dependency are read along their columns (a load takes 512 bytes of one; 16 consecutive
// entries per thread touched 32 lines a load: FP64 of order 2000, 79 -> 53 us) and turned in shared
// memory by the warp that reads them, so that every sum keeps its order.
constexpr int kTurnGroup = 18;  // 16 rows and 2 of padding: 16-byte reads of the four groups and two columns
constexpr int kTurnLd = 4 * kTurnGroup;  // meet in no bank
__device__ __forceinline__ constexpr int turned(int row) { return row + 2 * (row >> 4); }

__device__ __forceinline__ void turn_tile(double (*W)[kTurnLd], const double (&l)[8][2], double (&lt)[16]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < 8; ++e) *reinterpret_cast<double2*>(&W[e][turned(2 * lane)]) = make_double2(l[e][0], l[e][1]);
  __syncwarp();
#pragma unroll
  for (int u = 0; u < 16; u += 2) {
    const double2 v = *reinterpret_cast<const double2*>(&W[lane >> 2][(lane & 3) * kTurnGroup + u]);
    lt[u] = v.x;
    lt[u + 1] = v.y;
  }
  __syncwarp();
}
// acc += l . v over this lane's 16 rows, v in turned() order
__device__ __forceinline__ double dot_rows(const double (&l)[16], const double* v, double acc) {
  const double* p = v + (threadIdx.x & 3) * kTurnGroup;
#pragma unroll
  for (int u = 0; u < 16; u += 2) {
    const double2 x = *reinterpret_cast<const double2*>(p + u);
    acc += l[u] * x.x;
    acc += l[u + 1] * x.y;
  }
  return acc;
}

template <class T>
__global__ void __launch_bounds__(256, 1) k_trsv_bwd(const T* __restrict__ M, int ld, const T* __restrict__ Linv, int nb,
                                                  double* z, double* Y, double* X, int* err) {
  __shared__ __align__(16) double W[8][8][kTurnLd];
  __shared__ __align__(16) double xs[2][kTurnLd];
  __shared__ __align__(16) double rhs[kTurnLd];
  __shared__ double part[4][kNB];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, c = warp * 8 + (lane >> 2), g = lane & 3;
  for (int q = blockIdx.x; q < nb; q += gridDim.x) {
    const int i = nb - 1 - q;
    // this thread's entries of Linv_ii and of L_{i+1,i} (the last dependency), loaded before any wait
    double li[16], lp[16];
    load16(Linv + static_cast<int64_t>(i) * kNB * kNB + c * kNB + g * 16, li);  // rows 16g .. of column c of Linv_ii
    if (i + 1 < nb) load16(M + static_cast<int64_t>(i * kNB + c) * ld + g * 16 + (i + 1) * kNB, lp);
    double yi = 0.0;
    if (t < kNB) {
      yi = Y[i * kNB + t];
      Y[i * kNB + t] = __longlong_as_double(static_cast<long long>(kUnset));
    }
    double acc = 0.0;
    const T* tile = M + static_cast<int64_t>(i * kNB + warp * 8) * ld + lane * 2;
    double l[8][2];
    if (nb - 1 > i + 1) {
#pragma unroll
      for (int e = 0; e < 8; ++e) load2(tile + static_cast<int64_t>(e) * ld + (nb - 1) * kNB, l[e]);
    }
    for (int j = nb - 1; j > i + 1; --j) {  // blocks nb-1 down to i+2
      double lt[16];
      turn_tile(W[warp], l, lt);
      if (j - 1 > i + 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) load2(tile + static_cast<int64_t>(e) * ld + (j - 1) * kNB, l[e]);
      }
      if (t < kNB) xs[j & 1][turned(t)] = wait_value(X + j * kNB + t, err);
      __syncthreads();
      acc = dot_rows(lt, xs[j & 1], acc);
    }
    if (i + 1 < nb) {
      double(&xl)[kTurnLd] = xs[(i + 1) & 1];
      if (t < kNB) xl[turned(t)] = wait_value(X + (i + 1) * kNB + t, err);
      __syncthreads();
      acc = dot_rows(lp, xl, acc);
    }
    part[g][c] = acc;
    __syncthreads();
    if (t < kNB) rhs[turned(t)] = yi - (part[0][t] + part[1][t] + part[2][t] + part[3][t]);
    __syncthreads();
    // x_c = sum_r Linv[r][c] rhs[r]
    part[g][c] = dot_rows(li, rhs, 0.0);
    __syncthreads();
    if (t < kNB) {
      const double v = part[0][t] + part[1][t] + part[2][t] + part[3][t];
      publish_value(X + i * kNB + t, v);
      z[i * kNB + t] = v;
    }
    __syncthreads();
  }
}

// Co-resident blocks of the cooperative solves, per device (queried once per device).
int dataflow_grid(int nb) {
  static int max_blocks[kMaxDevices] = {};
  int dev = 0;
  SOV_CUDA(cudaGetDevice(&dev));
  if (dev >= kMaxDevices) throw std::runtime_error("dense solve: device index beyond the supported 64");
  once_per_device((const void*)&max_blocks, [&] {
    int sms = 0, per_sm = 1 << 30;
    SOV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    for (const void* k : {(const void*)k_trsv_fwd<double>, (const void*)k_trsv_bwd<double>, (const void*)k_trsv_fwd<float>,
                          (const void*)k_trsv_bwd<float>}) {
      int n = 0;
      SOV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 256, 0));
      per_sm = std::min(per_sm, n);
    }
    max_blocks[dev] = std::max(1, sms * std::max(1, per_sm));
  });
  std::lock_guard<std::mutex> g(once_mutex());  // the write above happened under this lock
  return std::min(nb, max_blocks[dev]);
}

template <class T>
void dense_solve(const DenseSystem<T>& s, double* z, int* err, cudaStream_t st, int* launches) {
  const int grid = dataflow_grid(s.nb);
  const T* M = s.M;
  const T* Linv = s.Linv;
  int ld = s.mp, nb = s.nb;
  double *Y = s.chain, *X = s.chain + s.mp;
  const double* zc = z;
  void* args1[] = {(void*)&M, (void*)&ld, (void*)&Linv, (void*)&nb, (void*)&zc, (void*)&Y, (void*)&X, (void*)&err};
  SOV_CUDA(cudaLaunchCooperativeKernel((const void*)k_trsv_fwd<T>, dim3(grid), dim3(256), args1, 0, st));
  void* args2[] = {(void*)&M, (void*)&ld, (void*)&Linv, (void*)&nb, (void*)&z, (void*)&Y, (void*)&X, (void*)&err};
  SOV_CUDA(cudaLaunchCooperativeKernel((const void*)k_trsv_bwd<T>, dim3(grid), dim3(256), args2, 0, st));
  if (launches) *launches += 2;
}

// ---------------------------------------------------------------------------------------------
// Forward substitution with many right-hand sides: Y <- L^-1 Y (Y column-major, nrhs columns).
// One CTA per (row block i, tile of kRhsTile columns), taken in ticket order with i slowest, so an
// item only waits (acquire flag, bounded) for items of lower tickets, which run or have run; the
// tiles are independent chains of nb blocks. Latency of a chain step bounds it, not arithmetic:
// the rows of A used to go through a forward and a backward launch each, 33 us a row (portfolio QP of
// 25 rows, order 448: 16.8 -> 7.3 ms per solve of 12 iterations).
// ---------------------------------------------------------------------------------------------
// Both tiles of L a chain step needs are in shared memory (or on their way in registers) before its flag
// is awaited; read from L2 after it they were half of the chain: 62.6 -> 32.3 us a launch.
constexpr int kRhsTile = 8;  // 8 rather than 32 columns: a chain step's arithmetic shrinks with it (104 -> 59 us)

__global__ void __launch_bounds__(256) k_trsm_fwd(const double* __restrict__ M, int ld, const double* __restrict__ Linv,
                                                  int nb, double* Y, int ldy, int nrhs, unsigned* flags, int* err) {
  extern __shared__ __align__(16) unsigned char trsm_raw[];
  double(*Ls)[kNB] = reinterpret_cast<double(*)[kNB]>(trsm_raw);  // [column][row] of L_ij
  double(*Lis)[kNB] = Ls + kNB;                                   // and of Linv_ii
  __shared__ __align__(16) double ys[kRhsTile][kNB];
  __shared__ unsigned item_s;
  __shared__ int ok_s;
  const int t = threadIdx.x, r = t & (kNB - 1), g = t >> 6;
  const int tiles = (nrhs + kRhsTile - 1) / kRhsTile;
  if (t == 0) item_s = atomicAdd(flags + nb * tiles, 1u);
  __syncthreads();
  const int i = static_cast<int>(item_s) / tiles, tile = static_cast<int>(item_s) % tiles;
  const int c0 = tile * kRhsTile, cols = min(kRhsTile, nrhs - c0);
  constexpr int C = kRhsTile / 4;  // columns per thread
  double acc[C] = {}, yi[C], next[16];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int cc = g * C + c;
    yi[c] = cc < cols ? Y[static_cast<int64_t>(c0 + cc) * ldy + i * kNB + r] : 0.0;
  }
  const double* Li = Linv + static_cast<int64_t>(i) * kNB * kNB + r;
#pragma unroll
  for (int u = 0; u < 16; ++u) Lis[g + 4 * u][r] = Li[(g + 4 * u) * kNB];
  const double* Lij = M + static_cast<int64_t>(g) * ld + i * kNB + r;
  if (i > 0) {
#pragma unroll
    for (int u = 0; u < 16; ++u) next[u] = Lij[static_cast<int64_t>(4 * u) * ld];
  }
  for (int j = 0; j < i; ++j) {
#pragma unroll
    for (int u = 0; u < 16; ++u) Ls[g + 4 * u][r] = next[u];
    if (j + 1 < i) {
#pragma unroll
      for (int u = 0; u < 16; ++u) next[u] = Lij[static_cast<int64_t>((j + 1) * kNB + 4 * u) * ld];
    }
    if (t == 0) ok_s = wait_flag(flags + tile * nb + j, 1u);
    __syncthreads();
    if (!ok_s && t == 0) atomicExch(err, 1);
#pragma unroll
    for (int u = 0; u < C; ++u) {
      const int c = g + 4 * u;
      ys[c][r] = c < cols ? __ldcg(Y + static_cast<int64_t>(c0 + c) * ldy + j * kNB + r) : 0.0;
    }
    __syncthreads();
#pragma unroll 16
    for (int k = 0; k < kNB; k += 2) {
      const double l0 = Ls[k][r], l1 = Ls[k + 1][r];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const double2 y2 = *reinterpret_cast<const double2*>(&ys[g * C + c][k]);
        acc[c] += l0 * y2.x;
        acc[c] += l1 * y2.y;
      }
    }
    __syncthreads();
  }
  // Y_i <- L_ii^-1 (Y_i - acc)
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int cc = g * C + c;
    ys[cc][r] = yi[c] - acc[c];
    acc[c] = 0.0;
  }
  __syncthreads();
#pragma unroll 16
  for (int k = 0; k < kNB; k += 2) {
    const double l0 = Lis[k][r], l1 = Lis[k + 1][r];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const double2 y2 = *reinterpret_cast<const double2*>(&ys[g * C + c][k]);
      acc[c] += l0 * y2.x;
      acc[c] += l1 * y2.y;
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int cc = g * C + c;
    if (cc < cols) Y[static_cast<int64_t>(c0 + cc) * ldy + i * kNB + r] = acc[c];
  }
  __threadfence();
  __syncthreads();
  if (t == 0) st_release(flags + tile * nb + i, 1u);
}

size_t dense_forward_flags(int nb, int nrhs) {
  return static_cast<size_t>(nb) * ceil_div(std::max(1, nrhs), kRhsTile) + 1;
}

void dense_forward_multi(const DenseSystem<double>& s, double* Y, int ldy, int nrhs, unsigned* flags, int* err,
                         cudaStream_t st, int* launches) {
  if (nrhs <= 0) return;
  SOV_CUDA(cudaMemsetAsync(flags, 0, sizeof(unsigned) * dense_forward_flags(s.nb, nrhs), st));
  constexpr int smem = 2 * kNB * kNB * sizeof(double);
  once_per_device((const void*)k_trsm_fwd, [&] {
    SOV_CUDA(cudaFuncSetAttribute(k_trsm_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  });
  k_trsm_fwd<<<s.nb * ceil_div(nrhs, kRhsTile), 256, smem, st>>>(s.M, s.mp, s.Linv, s.nb, Y, ldy, nrhs, flags, err);
  SOV_LAUNCH_CHECK();
  if (launches) *launches += 1;
}

// explicit instantiations
template void launch_assemble<double>(const AssemblyDev&, const double*, const double*, const double*,
                                     const uint8_t*, int, double, double*, double*, int, int, cudaStream_t);
template void launch_assemble<float>(const AssemblyDev&, const double*, const double*, const double*,
                                    const uint8_t*, int, double, float*, double*, int, int, cudaStream_t);
template void launch_dense_clear<double>(double*, int, int, cudaStream_t);
template void launch_dense_clear<float>(float*, int, int, cudaStream_t);
template void dense_potrf_block<double>(const DenseSystem<double>&, int, cudaStream_t);
template void dense_potrf_block<float>(const DenseSystem<float>&, int, cudaStream_t);
template void dense_cholesky<double>(const DenseSystem<double>&, cudaStream_t, int*);
template void dense_solve<double>(const DenseSystem<double>&, double*, int*, cudaStream_t, int*);
template void dense_solve<float>(const DenseSystem<float>&, double*, int*, cudaStream_t, int*);

}  // namespace sov
