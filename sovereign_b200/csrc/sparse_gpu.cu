// sparse_gpu.cu -- numeric sparse L D L' and its solves on the GPU (see sparse_gpu.cuh).
#include "sparse_gpu.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <numeric>
#include <stdexcept>
#include <string>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace sov {
namespace {

constexpr int kSparseThreads = 256;
constexpr int kCtaThreads = 1024;  // the one-CTA forms

// Threads of a walk over the levels and the barrier between them: the whole grid, or one CTA.
struct GridWalk {
  cg::grid_group g;
  __device__ GridWalk() : g(cg::this_grid()) {}
  __device__ int rank() const { return static_cast<int>(g.thread_rank()); }
  __device__ int size() const { return static_cast<int>(g.size()); }
  __device__ void sync() const { g.sync(); }
};
struct CtaWalk {
  __device__ int rank() const { return static_cast<int>(threadIdx.x); }
  __device__ int size() const { return static_cast<int>(blockDim.x); }
  __device__ void sync() const { __syncthreads(); }
};

__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Per level: the pivots of its columns (one thread each), then its rank-1 updates, one warp per
// piece: lane l sums the piece's terms l, l + 32, ... and the warp adds the 32 partial sums in a
// fixed tree; a run cut into pieces is finished by its combine step (deterministic either way).
// After the last level the rows of L are left scaled for the one-CTA forward solve (fval = L~ / D by
// rows; the grid form gains nothing from it).
template <class Walk>
__device__ __forceinline__ void factor_levels(const SparseDev& s) {
  const Walk g;
  const int rank = g.rank(), size = g.size();
  const int lane = threadIdx.x & 31, warp = rank >> 5, warps = size >> 5;
  int drops = 0, bad = 0;
  for (int h = 0; h < s.levels; ++h) {
    for (int q = s.lvl_ptr[h] + rank; q < s.lvl_ptr[h + 1]; q += size) {
      const int k = s.lvl_col[q];
      const double p = s.V[k];
      const double sg = s.sign ? static_cast<double>(s.sign[k]) : 1.0;
      const bool finite = fabs(p) <= 1.7976931348623157e308;
      const bool drop = !(finite && sg * p > s.drop_tol * fabs(s.diag[k]));
      bad |= !finite;
      drops += drop;
      s.inv_d[k] = 1.0 / (drop ? sg * 1e128 : p);
    }
    g.sync();
    for (int q = s.fpiece_lvl[h] + rank; q < s.fwarp_lvl[h]; q += size) {  // short pieces: a thread each
      const int4 pc = s.fpiece[q];
      double acc = 0.0;
      for (int u = pc.x; u < pc.y; ++u) acc += s.V[s.m + s.up_a[u]] * s.V[s.m + s.up_b[u]] * s.inv_d[s.up_col[u]];
      if (pc.w < 0) s.V[pc.z] -= acc;
      else s.partial[pc.w] = acc;
    }
    for (int q = s.fwarp_lvl[h] + warp; q < s.fpiece_lvl[h + 1]; q += warps) {
      const int4 pc = s.fpiece[q];
      double acc = 0.0;
      for (int u = pc.x + lane; u < pc.y; u += 32)
        acc += s.V[s.m + s.up_a[u]] * s.V[s.m + s.up_b[u]] * s.inv_d[s.up_col[u]];
      acc = warp_total(acc);
      if (lane == 0) {
        if (pc.w < 0) s.V[pc.z] -= acc;
        else s.partial[pc.w] = acc;
      }
    }
    if (s.fcomb_lvl[h + 1] > s.fcomb_lvl[h]) {  // uniform: every thread reads the same bounds
      g.sync();
      for (int c = s.fcomb_lvl[h] + rank; c < s.fcomb_lvl[h + 1]; c += size) {
        const int4 cb = s.fcomb[c];
        double t = 0.0;
        for (int k = 0; k < cb.z; ++k) t += s.partial[cb.y + k];
        s.V[cb.x] -= t;
      }
    }
    g.sync();
  }
  for (int t = rank; s.fval && t < s.nnz; t += size) s.fval[t] = s.V[s.m + s.row_pos[t]] * s.inv_d[s.row_col[t]];
  if (drops) atomicAdd(s.drop_count, drops);
  if (bad) atomicExch(s.fail, 1);
}

__global__ void __launch_bounds__(kSparseThreads) k_sparse_factor(SparseDev s) { factor_levels<GridWalk>(s); }
__global__ void __launch_bounds__(kCtaThreads, 1) k_sparse_factor_cta(SparseDev s) { factor_levels<CtaWalk>(s); }

// L D L' x = z: forward y_k = z_k - sum_j L~_kj (1/D_j) y_j (row k of L, descendants: earlier
// levels), backward x_k = (1/D_k) (y_k - sum_i L~_ik x_i) (column k, ancestors: later levels);
// one warp per piece, partial sums added in a fixed tree, long rows and columns through their
// combine steps
__global__ void __launch_bounds__(kSparseThreads) k_sparse_solve(SparseDev s, double* z, const int* run) {
  if (run && !*run) return;  // written by an earlier launch: every block takes the same exit
  cg::grid_group g = cg::this_grid();
  const int rank = static_cast<int>(g.thread_rank()), size = static_cast<int>(g.size());
  const int lane = threadIdx.x & 31, warp = rank >> 5, warps = size >> 5;
  for (int k = rank; k < s.m; k += size) s.work[k] = z[s.perm[k]];
  g.sync();
  for (int h = 0; h < s.levels; ++h) {
    for (int q = s.lpiece_lvl[h] + rank; q < s.lwarp_lvl[h]; q += size) {
      const int4 pc = s.lpiece[q];
      double acc = 0.0;
      for (int t = pc.x; t < pc.y; ++t) acc += s.V[s.m + s.row_pos[t]] * s.inv_d[s.row_col[t]] * s.work[s.row_col[t]];
      if (pc.w < 0) s.work[pc.z] -= acc;
      else s.partial[pc.w] = acc;
    }
    for (int q = s.lwarp_lvl[h] + warp; q < s.lpiece_lvl[h + 1]; q += warps) {
      const int4 pc = s.lpiece[q];
      double acc = 0.0;
      for (int t = pc.x + lane; t < pc.y; t += 32)
        acc += s.V[s.m + s.row_pos[t]] * s.inv_d[s.row_col[t]] * s.work[s.row_col[t]];
      acc = warp_total(acc);
      if (lane == 0) {
        if (pc.w < 0) s.work[pc.z] -= acc;
        else s.partial[pc.w] = acc;
      }
    }
    if (s.lcomb_lvl[h + 1] > s.lcomb_lvl[h]) {
      g.sync();
      for (int c = s.lcomb_lvl[h] + rank; c < s.lcomb_lvl[h + 1]; c += size) {
        const int4 cb = s.lcomb[c];
        double t = 0.0;
        for (int k = 0; k < cb.z; ++k) t += s.partial[cb.y + k];
        s.work[cb.x] -= t;
      }
    }
    g.sync();
  }
  for (int h = s.levels - 1; h >= 0; --h) {
    for (int q = s.upiece_lvl[h] + rank; q < s.uwarp_lvl[h]; q += size) {
      const int4 pc = s.upiece[q];
      double acc = 0.0;
      for (int p = pc.x; p < pc.y; ++p) acc += s.V[s.m + p] * s.work[s.li[p]];
      if (pc.w < 0) s.work[pc.z] = (s.work[pc.z] - acc) * s.inv_d[pc.z];
      else s.partial[pc.w] = acc;
    }
    for (int q = s.uwarp_lvl[h] + warp; q < s.upiece_lvl[h + 1]; q += warps) {
      const int4 pc = s.upiece[q];
      double acc = 0.0;
      for (int p = pc.x + lane; p < pc.y; p += 32) acc += s.V[s.m + p] * s.work[s.li[p]];
      acc = warp_total(acc);
      if (lane == 0) {
        if (pc.w < 0) s.work[pc.z] = (s.work[pc.z] - acc) * s.inv_d[pc.z];
        else s.partial[pc.w] = acc;
      }
    }
    if (s.ucomb_lvl[h + 1] > s.ucomb_lvl[h]) {
      g.sync();
      for (int c = s.ucomb_lvl[h] + rank; c < s.ucomb_lvl[h + 1]; c += size) {
        const int4 cb = s.ucomb[c];
        double t = 0.0;
        for (int k = 0; k < cb.z; ++k) t += s.partial[cb.y + k];
        s.work[cb.x] = (s.work[cb.x] - t) * s.inv_d[cb.x];
      }
    }
    g.sync();
  }
  for (int k = rank; k < s.m; k += size) z[s.perm[k]] = s.work[k];
}

// The same solve on one CTA with the right-hand side in shared memory: a barrier between levels is
// a CTA barrier and a gather of it costs tens of cycles, where the grid form pays a grid barrier and
// dependent L2 loads per level (4.4 us a level each way). The pieces of level h + 2 and the terms of
// level h + 1 are loaded while level h is summed, so only shared-memory accesses sit between two
// barriers. Same pieces, same order of every sum: bit-identical to the grid form.
constexpr int kAhead = 4;  // terms of a short piece loaded a level ahead

template <bool kForward>
__device__ __forceinline__ void sweep_levels(const SparseDev& s, double* work, const int* piece_lvl, const int* warp_lvl,
                                             const int* comb_lvl) {
  const int4* pieces = kForward ? s.lpiece : s.upiece;
  const int4* combs = kForward ? s.lcomb : s.ucomb;
  const double* vals = kForward ? s.fval : s.V + s.m;
  const int* idx = kForward ? s.row_col : s.li;
  const int tid = static_cast<int>(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  const int levels = s.levels;
  auto level = [&](int q) { return kForward ? q : levels - 1 - q; };
  auto load_piece = [&](int q) {  // this thread's first short piece of the q-th level walked
    if (q < levels) {
      const int h = level(q), at = piece_lvl[h] + tid;
      if (at < warp_lvl[h]) return pieces[at];
    }
    return make_int4(0, 0, -1, -1);
  };
  struct Terms {
    double v[kAhead], inv;
    int c[kAhead];
  };
  auto load_terms = [&](const int4& pc, Terms& t) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const bool on = pc.x + u < pc.y;
      t.v[u] = on ? vals[pc.x + u] : 0.0;
      t.c[u] = on ? idx[pc.x + u] : 0;
    }
    t.inv = !kForward && pc.z >= 0 && pc.w < 0 ? s.inv_d[pc.z] : 0.0;
  };
  auto apply = [&](const int4& pc, double acc, double inv) {
    if (pc.w >= 0) s.partial[pc.w] = acc;
    else if (kForward) work[pc.z] -= acc;
    else work[pc.z] = (work[pc.z] - acc) * inv;
  };
  int4 pc = load_piece(0), pn = load_piece(1);
  Terms tc, tn;
  load_terms(pc, tc);
  for (int q = 0; q < levels; ++q) {
    const int h = level(q);
    const int4 pf = load_piece(q + 2);
    load_terms(pn, tn);
    if (pc.z >= 0) {
      double acc = 0.0;
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (pc.x + u < pc.y) acc += tc.v[u] * work[tc.c[u]];
      for (int t = pc.x + kAhead; t < pc.y; ++t) acc += vals[t] * work[idx[t]];
      apply(pc, acc, tc.inv);
    }
    for (int at = piece_lvl[h] + tid + kCtaThreads; at < warp_lvl[h]; at += kCtaThreads) {
      const int4 p2 = pieces[at];
      double acc = 0.0;
      for (int t = p2.x; t < p2.y; ++t) acc += vals[t] * work[idx[t]];
      apply(p2, acc, kForward || p2.w >= 0 ? 0.0 : s.inv_d[p2.z]);
    }
    for (int at = warp_lvl[h] + warp; at < piece_lvl[h + 1]; at += kCtaThreads / 32) {
      const int4 p2 = pieces[at];
      double acc = 0.0;
      for (int t = p2.x + lane; t < p2.y; t += 32) acc += vals[t] * work[idx[t]];
      acc = warp_total(acc);
      if (lane == 0) apply(p2, acc, kForward || p2.w >= 0 ? 0.0 : s.inv_d[p2.z]);
    }
    if (comb_lvl[h + 1] > comb_lvl[h]) {  // uniform: every thread reads the same bounds
      __syncthreads();
      for (int c = comb_lvl[h] + tid; c < comb_lvl[h + 1]; c += kCtaThreads) {
        const int4 cb = combs[c];
        double t = 0.0;
        for (int k = 0; k < cb.z; ++k) t += s.partial[cb.y + k];
        if (kForward) work[cb.x] -= t;
        else work[cb.x] = (work[cb.x] - t) * s.inv_d[cb.x];
      }
    }
    __syncthreads();
    pc = pn;
    pn = pf;
    tc = tn;
  }
}

// work (m doubles) | six level arrays (levels + 1 ints each)
size_t cta_solve_smem(int m, int levels) {
  return sizeof(double) * static_cast<size_t>(m) + sizeof(int) * 6 * (static_cast<size_t>(levels) + 1);
}

__global__ void __launch_bounds__(kCtaThreads, 1) k_sparse_solve_cta(SparseDev s, double* z, const int* run) {
  if (run && !*run) return;
  extern __shared__ double sm[];
  double* work = sm;
  int* lv = reinterpret_cast<int*>(sm + s.m);
  const int L1 = s.levels + 1, tid = static_cast<int>(threadIdx.x);
  for (int h = tid; h < L1; h += kCtaThreads) {
    lv[h] = s.lpiece_lvl[h];
    lv[L1 + h] = h < s.levels ? s.lwarp_lvl[h] : 0;
    lv[2 * L1 + h] = s.lcomb_lvl[h];
    lv[3 * L1 + h] = s.upiece_lvl[h];
    lv[4 * L1 + h] = h < s.levels ? s.uwarp_lvl[h] : 0;
    lv[5 * L1 + h] = s.ucomb_lvl[h];
  }
  for (int k = tid; k < s.m; k += kCtaThreads) work[k] = z[s.perm[k]];
  __syncthreads();
  sweep_levels<true>(s, work, lv, lv + L1, lv + 2 * L1);
  sweep_levels<false>(s, work, lv + 3 * L1, lv + 4 * L1, lv + 5 * L1);
  for (int k = tid; k < s.m; k += kCtaThreads) z[s.perm[k]] = work[k];
}

template <class T>
T* put(std::vector<void*>& bufs, const std::vector<T>& h, cudaStream_t st) {
  T* p = nullptr;
  SOV_CUDA(cudaMalloc(&p, sizeof(T) * std::max<size_t>(1, h.size())));
  bufs.push_back(p);
  if (!h.empty()) SOV_CUDA(cudaMemcpyAsync(p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, st));
  return p;
}

}  // namespace

void SparseFactor::upload(const SparseSymbolic& s, int* drop_count, int* fail, double drop_tol, cudaStream_t st,
                          const std::vector<int8_t>* sign) {
  release();
  const int m = s.m, levels = s.levels();
  nnz_l_ = s.nnz_l;
  const SparseSchedule S = sparse_schedule(s);
  d_.m = m;
  d_.levels = levels;
  d_.V = put(bufs_, std::vector<double>(m + s.li.size(), 0.0), st);
  d_.diag = put(bufs_, std::vector<double>(m, 0.0), st);
  d_.inv_d = put(bufs_, std::vector<double>(m, 0.0), st);
  d_.nnz = static_cast<int>(s.li.size());
  d_.work = put(bufs_, std::vector<double>(m, 0.0), st);
  d_.perm = put(bufs_, s.perm, st);
  d_.lp = put(bufs_, s.lp, st);
  d_.li = put(bufs_, s.li, st);
  d_.lvl_ptr = put(bufs_, s.lvl_ptr, st);
  d_.lvl_col = put(bufs_, s.lvl_col, st);
  static_assert(sizeof(SparsePiece) == sizeof(int4) && sizeof(SparseCombine) == sizeof(int4), "piece layout");
  auto put4 = [&](const auto& v) { return reinterpret_cast<const int4*>(put(bufs_, v, st)); };
  d_.fpiece = put4(S.factor.piece);
  d_.fpiece_lvl = put(bufs_, S.factor.piece_lvl, st);
  d_.fwarp_lvl = put(bufs_, S.factor.warp_lvl, st);
  d_.fcomb = put4(S.factor.comb);
  d_.fcomb_lvl = put(bufs_, S.factor.comb_lvl, st);
  d_.lpiece = put4(S.forward.piece);
  d_.lpiece_lvl = put(bufs_, S.forward.piece_lvl, st);
  d_.lwarp_lvl = put(bufs_, S.forward.warp_lvl, st);
  d_.lcomb = put4(S.forward.comb);
  d_.lcomb_lvl = put(bufs_, S.forward.comb_lvl, st);
  d_.upiece = put4(S.backward.piece);
  d_.upiece_lvl = put(bufs_, S.backward.piece_lvl, st);
  d_.uwarp_lvl = put(bufs_, S.backward.warp_lvl, st);
  d_.ucomb = put4(S.backward.comb);
  d_.ucomb_lvl = put(bufs_, S.backward.comb_lvl, st);
  d_.partial = put(bufs_, std::vector<double>(std::max(1, std::max(S.factor_slots, S.solve_slots)), 0.0), st);
  d_.up_col = put(bufs_, S.up_col, st);
  d_.up_a = put(bufs_, S.up_a, st);
  d_.up_b = put(bufs_, S.up_b, st);
  d_.row_pos = put(bufs_, S.row_pos, st);
  d_.row_col = put(bufs_, S.row_col, st);
  d_.drop_count = drop_count;
  d_.fail = fail;
  d_.drop_tol = drop_tol;
  d_.sign = nullptr;
  std::vector<int8_t> sign_elim;
  if (sign) {
    sign_elim.resize(m);
    for (int k = 0; k < m; ++k) sign_elim[k] = (*sign)[s.perm[k]];
    d_.sign = put(bufs_, sign_elim, st);
  }
  SOV_CUDA(cudaStreamSynchronize(st));  // the host vectors above go out of scope
  int dev = 0, sms = 0, per_sm = 0;
  SOV_CUDA(cudaGetDevice(&dev));
  SOV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  SOV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sparse_factor, kSparseThreads, 0));
  int per_sm2 = 0;
  SOV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm2, k_sparse_solve, kSparseThreads, 0));
  // one CTA per SM: most levels hold few columns, and a grid barrier costs more with more CTAs
  grid_ = std::max(1, sms * std::min(1, std::min(per_sm, per_sm2)));
  int smem_max = 0;
  SOV_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t smem = cta_solve_smem(m, levels);
  cta_factor_ = factor_on_one_cta(m, levels, static_cast<long long>(S.up_col.size()));
  cta_solve_ = smem <= static_cast<size_t>(smem_max) && solve_on_one_cta(m, levels, nnz_l_);
  // SOVEREIGN_SPARSE_WALK=grid|cta: one form for every matrix it can take (the tests compare the two)
  if (const char* e = std::getenv("SOVEREIGN_SPARSE_WALK")) {
    const bool cta = std::string(e) == "cta";
    if (cta || std::string(e) == "grid") {
      cta_factor_ = cta;
      cta_solve_ = cta && smem <= static_cast<size_t>(smem_max);
    }
  }
  if (cta_solve_) {
    d_.fval = put(bufs_, std::vector<double>(s.li.size(), 0.0), st);
    SOV_CUDA(cudaStreamSynchronize(st));
    once_per_device((const void*)k_sparse_solve_cta, [&] {
      SOV_CUDA(cudaFuncSetAttribute(k_sparse_solve_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    });
  }
}

void SparseFactor::release() {
  for (void* p : bufs_) cudaFree(p);
  bufs_.clear();
  d_ = SparseDev{};
}

void SparseFactor::factor(cudaStream_t st, int* launches) {
  SparseDev d = d_;
  if (launches) *launches += 1;
  if (cta_factor_) {
    k_sparse_factor_cta<<<1, kCtaThreads, 0, st>>>(d);
    SOV_LAUNCH_CHECK();
    return;
  }
  void* args[] = {&d};
  SOV_CUDA(cudaLaunchCooperativeKernel((const void*)k_sparse_factor, dim3(grid_), dim3(kSparseThreads), args, 0, st));
}

void SparseFactor::solve(double* z, cudaStream_t st, int* launches, const int* run) {
  SparseDev d = d_;
  if (launches) *launches += 1;
  if (cta_solve_) {
    k_sparse_solve_cta<<<1, kCtaThreads, cta_solve_smem(d.m, d.levels), st>>>(d, z, run);
    SOV_LAUNCH_CHECK();
    return;
  }
  void* args[] = {&d, &z, &run};
  SOV_CUDA(cudaLaunchCooperativeKernel((const void*)k_sparse_solve, dim3(grid_), dim3(kSparseThreads), args, 0, st));
}

}  // namespace sov
