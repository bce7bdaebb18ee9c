// The Coupled solve's coarse levels for sm_100a (compiled with --fmad=false,
// IEEE division): Galerkin operators, smoother bound, residual, damped
// block-Jacobi sweep and transfers of src/kutta/kernels/fv_coupled.kern.h, each
// sum in the reference's order.
//
// These levels are latency-bound: 10^2 to 10^5 rows of 7 to 150 entries whose
// operator sits in L2. Two rules follow, and both keep the order of every sum:
// - what is independent runs in parallel threads: a block loads its rows'
//   entries coalesced and forms their products in shared memory, then four
//   threads per row add one component (u, v, w, p) each; a Galerkin entry is
//   eight threads, one per coefficient, over a list of its contributions
//   built once at setup;
// - what a solve does not change between two kernels (pattern, entries, block
//   inverses) is loaded before the wait for the previous kernel.
#include <cuda_runtime.h>

#include <atomic>

#include "coupled_kernels.hpp"
#include "coupled_rows.cuh"

namespace kb2 {
namespace {

using namespace dev;

__device__ __forceinline__ float component(const float4& v, int k) {
  return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}
__device__ __forceinline__ float4 plus(float4 a, const float4& b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
  a.w += b.w;
  return a;
}

// An entry's products with its column's unknowns (fv_coupled.kern.h:376-392).
__device__ __forceinline__ float4 entry_terms(const float4& e, const float4& h, const float4& x) {
  return make_float4(e.x * x.x + e.y * x.w, e.x * x.y + e.z * x.w, e.x * x.z + e.w * x.w,
                     h.y * x.x + h.z * x.y + h.w * x.z + h.x * x.w);
}

enum class Pass { Residual, Smooth, SmoothProlonged };

// Rows [row0, row0 + kRows) of a level by the kThreads threads of a block, four
// threads per row: the residual b - J x, or the sweep from x (from x +
// coarse[aggregate], the prolongation, in the first post-sweep). The operator
// is loaded before the wait for the previous kernel.
template <int kThreads, int kRows, int kPer, Pass kPass>
__global__ void __launch_bounds__(kThreads) k_cpl_coarse_rows(
    CoupledLevel l, const float4* __restrict__ x, const float4* __restrict__ b,
    float4* __restrict__ out, float omega, const int* __restrict__ aggregate,
    const float4* __restrict__ coarse) {
  constexpr int kStage = kThreads * kPer;
  __shared__ float4 staged[kStage];
  const int row0 = blockIdx.x * kRows;
  constexpr bool kSmooth = kPass != Pass::Residual, kProlong = kPass == Pass::SmoothProlonged;
  static_assert(4 * kRows <= kThreads, "four threads per row");
  const std::size_t N = l.n;
  const int tid = threadIdx.x, part = tid & 3;
  const int first = l.rows[row0], last = l.rows[min(l.n, row0 + kRows)];
  const int i = row0 + (tid >> 2);
  const bool owner = (tid >> 2) < kRows && i < l.n;
  const int begin = owner ? l.rows[i] : 0, end = owner ? l.rows[i + 1] : 0;
  const int diag = owner ? l.diag[i] : 0;
  float4 ek = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hk = ek;
  float own = 0.0f, inverse = 0.0f, hu = 0.0f, hv = 0.0f, hw = 0.0f, schur = 1.0f;
  int group = -1;
  if (owner) {
    ek = l.entry[2 * static_cast<std::size_t>(diag)];
    hk = l.entry[2 * static_cast<std::size_t>(diag) + 1];
    if (part < 3) own = l.d[part * N + i];
    if (kSmooth) {
      if (part < 3) inverse = l.d[(4 + part) * N + i];
      hu = l.d[7 * N + i];
      hv = l.d[8 * N + i];
      hw = l.d[9 * N + i];
      schur = l.d[10 * N + i];
    }
    if (kProlong) group = aggregate[i];
  }
  int c[kPer], g[kPer];
  float4 e[kPer], h[kPer];
  const auto load = [&](int base) {
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int j = base + tid + k * kThreads;
      c[k] = j < last ? l.cols[j] : -1;
      if (c[k] < 0) continue;
      e[k] = l.entry[2 * static_cast<std::size_t>(j)];
      h[k] = l.entry[2 * static_cast<std::size_t>(j) + 1];
      if (kProlong) g[k] = aggregate[c[k]];
    }
  };
  load(first);
  pdl_entry();
  float4 xi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float y = 0.0f, right = 0.0f;
  if (owner) {
    xi = x[i];
    if (kProlong) xi = plus(xi, coarse[group]);
    right = reinterpret_cast<const float*>(b)[4 * static_cast<std::size_t>(i) + part];
    y = part == 3 ? hk.x * xi.w + hk.y * xi.x + hk.z * xi.y + hk.w * xi.z
                  : own * component(xi, part) + component(ek, part + 1) * xi.w;
  }
  const float* terms = reinterpret_cast<const float*>(staged) + part;
  for (int base = first; base < last; base += kStage) {
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (c[k] < 0) continue;
      float4 xm = x[c[k]];
      if (kProlong) xm = plus(xm, coarse[g[k]]);
      staged[tid + k * kThreads] = entry_terms(e[k], h[k], xm);
    }
    __syncthreads();
    if (base + kStage < last) load(base + kStage);
    const int to = min(end, base + kStage) - base;
#pragma unroll 4
    for (int j = max(begin, base) - base; j < to; ++j)
      if (base + j != diag) y += terms[4 * j];
    __syncthreads();
  }
  const float r = right - y;
  if constexpr (!kSmooth) {
    if (owner) reinterpret_cast<float*>(out)[4 * static_cast<std::size_t>(i) + part] = r;
    return;
  }
  const int lane = tid & 28;
  const float ru = __shfl_sync(0xffffffffu, r, lane), rv = __shfl_sync(0xffffffffu, r, lane + 1),
              rw = __shfl_sync(0xffffffffu, r, lane + 2), rp = __shfl_sync(0xffffffffu, r, lane + 3);
  if (!owner) return;
  // The block solve (block_solve), one component per thread.
  const float p = (rp - hu * ru - hv * rv - hw * rw) / schur;
  const float step = part == 3 ? p : inverse * (r - component(ek, part + 1) * p);
  reinterpret_cast<float*>(out)[4 * static_cast<std::size_t>(i) + part] =
      component(xi, part) + omega * step;
}

// One damped block-Jacobi update from zero of the row whose right-hand side
// component the thread holds; all 32 lanes of the warp call it.
__device__ __forceinline__ float zero_sweep(const CoupledLevel& l, int i, int part, bool owner,
                                            float r, float omega) {
  const std::size_t N = l.n;
  const int lane = threadIdx.x & 28;
  const float ru = __shfl_sync(0xffffffffu, r, lane), rv = __shfl_sync(0xffffffffu, r, lane + 1),
              rw = __shfl_sync(0xffffffffu, r, lane + 2), rp = __shfl_sync(0xffffffffu, r, lane + 3);
  if (!owner) return 0.0f;
  const float p =
      (rp - l.d[7 * N + i] * ru - l.d[8 * N + i] * rv - l.d[9 * N + i] * rw) / l.d[10 * N + i];
  if (part == 3) return 0.0f + omega * p;
  const float e = reinterpret_cast<const float*>(l.entry)[8 * static_cast<std::size_t>(l.diag[i]) +
                                                          part + 1];
  return 0.0f + omega * (l.d[(4 + part) * N + i] * (r - e * p));
}

// fv_coupled.kern.h:401-416 with x = 0 (coupled_coarse_smooth, first).
__global__ void __launch_bounds__(kBlock) k_cpl_coarse_first(CoupledLevel l,
                                                             const float4* __restrict__ b,
                                                             float4* __restrict__ next,
                                                             float omega) {
  pdl_entry();
  const int at = blockIdx.x * kBlock + threadIdx.x, i = at >> 2, part = at & 3;
  const bool owner = i < l.n;
  const float r = owner ? reinterpret_cast<const float*>(b)[at] : 0.0f;
  const float x = zero_sweep(l, i, part, owner, r, omega);
  if (owner) reinterpret_cast<float*>(next)[at] = x;
}

// fv_coupled.kern.h:554-560: a member sum per component in member order, four
// threads per aggregate; with kFirst the coarse level's sweep from zero too.
template <bool kFirst>
__global__ void __launch_bounds__(kBlock) k_cpl_restrict(int nc, const int* __restrict__ offsets,
                                                         const int* __restrict__ members,
                                                         const float4* __restrict__ fine,
                                                         float4* __restrict__ coarse,
                                                         CoupledLevel l, float omega,
                                                         float4* __restrict__ next) {
  constexpr int kBatch = 8;
  const int at = blockIdx.x * kBlock + threadIdx.x, i = at >> 2, part = at & 3;
  const bool owner = i < nc;
  const int begin = owner ? offsets[i] : 0, end = owner ? offsets[i + 1] : 0;
  int m[kBatch];
#pragma unroll
  for (int k = 0; k < kBatch; ++k) m[k] = begin + k < end ? members[begin + k] : -1;
  pdl_entry();
  const float* f = reinterpret_cast<const float*>(fine) + part;
  float s = 0.0f;
  for (int j = begin; j < end; j += kBatch) {
    float v[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) v[k] = m[k] >= 0 ? f[4 * static_cast<std::size_t>(m[k])] : 0.0f;
#pragma unroll
    for (int k = 0; k < kBatch; ++k)
      if (j + k < end) {
        s += v[k];
        m[k] = j + kBatch + k < end ? members[j + kBatch + k] : -1;
      }
  }
  if (owner) reinterpret_cast<float*>(coarse)[at] = s;
  if constexpr (kFirst) {
    const float x = zero_sweep(l, i, part, owner, s, omega);
    if (owner) reinterpret_cast<float*>(next)[at] = x;
  }
}

// ---- Galerkin operators -------------------------------------------------------

// The entry of column `col` in coarse row `row` (fv_coupled.kern.h:418-422); a
// row's columns are sorted and unique.
__device__ __forceinline__ int entry_of(const int* __restrict__ rows, const int* __restrict__ cols,
                                        int row, int col) {
  int lo = rows[row];
  const int end = rows[row + 1];
  int hi = end;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cols[mid] < col)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < end && cols[lo] == col ? lo : -1;
}

// Appends term `value` to entry e's list: counts it, or (terms set) places it.
template <class Term>
__device__ __forceinline__ int add_term(const CoupledLevel& l, int e, Term value, int* count,
                                        Term* terms) {
  const int at = count[e]++;
  if (!terms) return 0;
  terms[l.term_at[e] + at] = value;
  return l.term_at[e] + at;
}

// One thread owns a coarse row and visits its contributions in the reference's
// order (fv_coupled.kern.h:424-524): members, then each one's faces or entries.
template <class Term>
__global__ void k_cpl_terms_fine(CoupledLevel l, CoupledTransfer t, int cells,
                                 const int* __restrict__ offsets, const int* __restrict__ adjacent,
                                 const int* __restrict__ faces, int* count, Term* terms,
                                 int* term_faces) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= l.n) return;
  for (int mm = t.offsets[i]; mm < t.offsets[i + 1]; ++mm) {
    const int q = t.members[mm];
    add_term(l, l.diag[i], ~static_cast<Term>(q), count, terms);
    int slot = 0;
    for (int j = offsets[q]; j < offsets[q + 1]; ++j) {
      const int other = adjacent[j];
      if (other < 0) continue;
      const int target = t.aggregate[other];
      const int e = target == i ? l.diag[i] : entry_of(l.rows, l.cols, i, target);
      if (e >= 0) {
        const int at = add_term(l, e, static_cast<Term>(slot) * cells + q, count, terms);
        if (terms) term_faces[at] = faces[j];
      }
      ++slot;
    }
  }
}
template <class Term>
__global__ void k_cpl_terms_coarse(CoupledLevel l, CoupledTransfer t, CoupledLevel f, int* count,
                                   Term* terms) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= l.n) return;
  for (int mm = t.offsets[i]; mm < t.offsets[i + 1]; ++mm) {
    const int row = t.members[mm];
    add_term(l, l.diag[i], ~static_cast<Term>(row), count, terms);
    for (int j = f.rows[row]; j < f.rows[row + 1]; ++j) {
      const int target = t.aggregate[f.cols[j]];
      const bool diagonal = j == f.diag[row];
      const int e = diagonal || target == i ? l.diag[i] : entry_of(l.rows, l.cols, i, target);
      if (e >= 0) add_term(l, e, 2 * static_cast<Term>(j) + (diagonal ? 1 : 0), count, terms);
    }
  }
}

// Where a contribution's coefficient lies. Fine level: the packed records of
// the ELL slot (the coefficients fv_coupled.kern.h:424-488 forms again: a, G, the
// negative Rhie-Chow coefficient, and H as share times face area).
template <class Term>
struct FromFine {
  CoupledFine op;
  const Term* terms;
  const int* faces;
  const float* cell;
  std::size_t cells;
  float wc;
  // Coefficient k of a term: a, gx, gy, gz, c, hx, hy, hz.
  // The face of a term comes from a list of its own beside the terms, so that
  // its load does not wait for the slot's link.
  __device__ __forceinline__ float value(Term term, int at, int k) const {
    if (k < 4) return reinterpret_cast<const float*>(op.edge)[4 * static_cast<std::size_t>(term) + k];
    const float* face =
        reinterpret_cast<const float*>(op.face) + 4 * static_cast<std::size_t>(faces[at]);
    return k == 4 ? -face[3] : op.edge_h[term] * face[k - 5];
  }
  // A member's own coefficient: u, v, w, c, gx, gy, gz, hx, hy, hz.
  __device__ __forceinline__ float own(int row, int k) const {
    const float v = cell[k * cells + row];
    return k < 4 ? v : wc * v;
  }
  // Whether a term adds to the momentum sums.
  static __device__ __forceinline__ bool momentum(Term) { return true; }
  static constexpr bool kOwnsAll = true;  // own() covers all ten sums
};
template <class Term>
struct FromLevel {
  CoupledLevel f;
  const Term* terms;
  __device__ __forceinline__ float value(Term term, int, int k) const {
    return reinterpret_cast<const float*>(f.entry)[8 * static_cast<std::size_t>(term >> 1) + k];
  }
  __device__ __forceinline__ float own(int row, int k) const {
    return f.d[k * static_cast<std::size_t>(f.n) + row];
  }
  static __device__ __forceinline__ bool momentum(Term term) { return (term & 1) == 0; }
  static constexpr bool kOwnsAll = false;  // only u, v, w
};

// Off-diagonal entries: eight threads each, one per coefficient, plain sums
// from zero in list order; a list's values are loaded four at a time.
template <class From>
__device__ __forceinline__ void sum_entry(const CoupledLevel& l, const From& from, int e, int k) {
  const int begin = l.term_at[e], end = l.term_at[e + 1];
  if (begin < end && from.terms[begin] < 0) return;  // a diagonal entry
  float sum = 0.0f;
  for (int j = begin; j < end; j += 4) {
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = j + u < end ? from.value(from.terms[j + u], j + u, k) : 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (j + u < end) sum += v[u];
  }
  reinterpret_cast<float*>(l.entry)[8 * static_cast<std::size_t>(e) + k] = sum;
}

// A row's diagonal: sixteen threads, ten of them with a compensated sum each
// (u, v, w, c, gx, gy, gz, hx, hy, hz).
template <class From>
__device__ __forceinline__ void sum_diagonal(const CoupledLevel& l, const From& from, int i, int k) {
  const int e = l.diag[i];
  // The coefficient of a term that sum k takes: a for the three momentum sums.
  const int which = k < 3 ? 0 : k == 3 ? 4 : k < 7 ? k - 3 : k - 2;
  Csum sum{0.0f, 0.0f};
  const int begin = l.term_at[e], end = l.term_at[e + 1];
  for (int j = begin; j < end; j += 4) {
    float v[4];
    bool add[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      add[u] = j + u < end;
      if (!add[u]) continue;
      const auto term = from.terms[j + u];
      if (term < 0) {
        add[u] = From::kOwnsAll || k < 3;
        if (add[u]) v[u] = from.own(static_cast<int>(~term), k);
      } else {
        add[u] = k >= 3 || From::momentum(term);
        if (add[u]) v[u] = from.value(term, j + u, which);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (add[u]) sum = csum_add(sum, v[u]);
  }
  float* entry = reinterpret_cast<float*>(l.entry) + 8 * static_cast<std::size_t>(e);
  if (k < 3)
    l.d[k * static_cast<std::size_t>(l.n) + i] = csum_value(sum);
  else
    entry[which] = csum_value(sum);
  if (k == 0) entry[0] = 0.0f;
}

// Galerkin product (fv_coupled.kern.h:424-524), every coefficient by its own
// thread: the diagonals' blocks first, their sums being the longest. A thread
// per coarse row, adding to its row's entries in memory one contribution
// after another, took 1.2 ms for the fine product of 884,736 hexes and 2.3 ms for
// the coarse ones.
template <class From>
__global__ void __launch_bounds__(kBlock) k_cpl_galerkin(CoupledLevel l, From from,
                                                         int diagonal_blocks) {
  pdl_entry();
  if (static_cast<int>(blockIdx.x) < diagonal_blocks) {
    const int at = blockIdx.x * kBlock + threadIdx.x, i = at >> 4, k = at & 15;
    if (i < l.n && k < 10) sum_diagonal(l, from, i, k);
  } else {
    const long long at =
        static_cast<long long>(blockIdx.x - diagonal_blocks) * kBlock + threadIdx.x;
    if (at < 8LL * l.nnz) sum_entry(l, from, static_cast<int>(at >> 3), static_cast<int>(at & 7));
  }
}

template <class From>
void galerkin(const CoupledLevel& l, const From& from, cudaStream_t s) {
  if (l.n <= 0) return;
  ++launch::counter;
  const int diagonals = (16 * l.n + kBlock - 1) / kBlock;
  const long long entries = (8LL * l.nnz + kBlock - 1) / kBlock;
  pdl(k_cpl_galerkin<From>, static_cast<unsigned>(diagonals + entries), kBlock, 0, s, l, from,
      diagonals);
}

// fv_coupled.kern.h:526-534 (coupled_coarse_gsum): into 3n of scratch, a thread
// per row and component.
__global__ void k_cpl_coarse_gsum(CoupledLevel l, float* __restrict__ r) {
  pdl_entry();
  const int at = blockIdx.x * blockDim.x + threadIdx.x, i = at >> 2, part = at & 3;
  if (i >= l.n || part == 3) return;
  const float* g = reinterpret_cast<const float*>(l.entry) + part + 1;
  float sum = 0.0f;
  const int end = l.rows[i + 1];
#pragma unroll 4
  for (int j = l.rows[i]; j < end; ++j) sum += fabsf(g[8 * static_cast<std::size_t>(j)]);
  r[part * static_cast<std::size_t>(l.n) + i] = sum;
}

// fv_coupled.kern.h:536-552 (coupled_coarse_schur): cs and the block inverse.
// Eight threads per row form the entries' terms, each reads them all by shuffle
// and adds them in order.
__global__ void k_cpl_coarse_schur(CoupledLevel l, const float* __restrict__ r) {
  pdl_entry();
  const std::size_t N = l.n;
  float* d = l.d;
  const int at = blockIdx.x * blockDim.x + threadIdx.x, i = at >> 3, part = at & 7;
  const int lane = threadIdx.x & 24;
  const unsigned mask = 0xffu << lane;
  if (i >= l.n) return;
  const int k = l.diag[i];
  float sum = 0.0f;
  const int end = l.rows[i + 1];
  for (int base = l.rows[i]; base < end; base += 8) {
    const int j = base + part;
    float term = 0.0f;
    if (j < end && j != k) {
      const int m = l.cols[j];
      const float4 h = l.entry[2 * static_cast<std::size_t>(j) + 1];
      term = fabsf(h.y) * r[m] / fmaxf(d[m], 1.0e-30f) +
             fabsf(h.z) * r[N + m] / fmaxf(d[N + m], 1.0e-30f) +
             fabsf(h.w) * r[2 * N + m] / fmaxf(d[2 * N + m], 1.0e-30f);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float next = __shfl_sync(mask, term, lane + u);
      if (base + u < end && base + u != k) sum += next;
    }
  }
  if (part != 0) return;
  d[3 * N + i] = sum;
  const float4 e = l.entry[2 * static_cast<std::size_t>(k)];
  const float4 h = l.entry[2 * static_cast<std::size_t>(k) + 1];
  const BlockInverse b =
      block_prepare(d[i], d[N + i], d[2 * N + i], e.y, e.z, e.w, h.y, h.z, h.w, h.x + sum);
  d[4 * N + i] = b.iu;
  d[5 * N + i] = b.iv;
  d[6 * N + i] = b.iw;
  d[7 * N + i] = b.hu;
  d[8 * N + i] = b.hv;
  d[9 * N + i] = b.hw;
  d[10 * N + i] = b.schur;
}

// ---- the small coarse levels in one launch --------------------------------------
//
// The V-cycle of the levels of at most kMaxRows rows and kMaxEntries entries, in
// one block of 512 threads, four per row: each sweep, residual, restriction
// and prolongation is a pass over the level with the arithmetic of the kernels
// above, separated by __syncthreads (no inter-block waits). The vectors lie in
// shared memory and the threads keep a level's operator in registers over all
// the passes of a visit, so a pass reads x, forms the terms and adds them.
constexpr int kTailThreads = 512, kTailPer = CoupledTail::kMaxEntries / kTailThreads;
static_assert(4 * CoupledTail::kMaxRows == kTailThreads, "four threads per row");

struct TailHeld {
  int column[kTailPer];
  float4 e[kTailPer], h[kTailPer];
  int begin, end, diag;
  float4 ek, hk;
  float own, inverse, hu, hv, hw, schur;
};
__device__ __forceinline__ void tail_hold(const CoupledLevel& l, TailHeld& t) {
  const std::size_t N = l.n;
  const int i = threadIdx.x >> 2, part = threadIdx.x & 3;
#pragma unroll
  for (int k = 0; k < kTailPer; ++k) {
    const int j = threadIdx.x + k * kTailThreads;
    t.column[k] = j < l.nnz ? l.cols[j] : -1;
    if (t.column[k] < 0) continue;
    t.e[k] = l.entry[2 * j];
    t.h[k] = l.entry[2 * j + 1];
  }
  t.begin = t.end = t.diag = 0;
  t.own = t.inverse = t.hu = t.hv = t.hw = 0.0f;
  t.schur = 1.0f;
  t.ek = t.hk = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (i >= l.n) return;
  t.begin = l.rows[i];
  t.end = l.rows[i + 1];
  t.diag = l.diag[i];
  t.ek = l.entry[2 * t.diag];
  t.hk = l.entry[2 * t.diag + 1];
  if (part < 3) {
    t.own = l.d[part * N + i];
    t.inverse = l.d[(4 + part) * N + i];
  }
  t.hu = l.d[7 * N + i];
  t.hv = l.d[8 * N + i];
  t.hw = l.d[9 * N + i];
  t.schur = l.d[10 * N + i];
}

// The residual, or the sweep from x (from zero when first), as level_rows.
__device__ __forceinline__ void tail_pass(int n, const TailHeld& t, const float4* x,
                                          const float4* b, float4* out, bool smooth, bool first,
                                          float omega, float4* staged) {
  const int i = threadIdx.x >> 2, part = threadIdx.x & 3;
  const bool owner = i < n;
  float r = owner ? reinterpret_cast<const float*>(b)[threadIdx.x] : 0.0f;
  float4 xi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (!first) {
    if (owner) xi = x[i];
#pragma unroll
    for (int k = 0; k < kTailPer; ++k)
      if (t.column[k] >= 0)
        staged[threadIdx.x + k * kTailThreads] = entry_terms(t.e[k], t.h[k], x[t.column[k]]);
    float y = part == 3 ? t.hk.x * xi.w + t.hk.y * xi.x + t.hk.z * xi.y + t.hk.w * xi.z
                        : t.own * component(xi, part) + component(t.ek, part + 1) * xi.w;
    __syncthreads();
    const float* terms = reinterpret_cast<const float*>(staged) + part;
#pragma unroll 8
    for (int j = t.begin; j < t.end; ++j)
      if (j != t.diag) y += terms[4 * j];
    r = r - y;
  }
  float value = r;
  if (smooth) {
    const int lane = threadIdx.x & 28;
    const float ru = __shfl_sync(0xffffffffu, r, lane),
                rv = __shfl_sync(0xffffffffu, r, lane + 1),
                rw = __shfl_sync(0xffffffffu, r, lane + 2),
                rp = __shfl_sync(0xffffffffu, r, lane + 3);
    const float p = (rp - t.hu * ru - t.hv * rv - t.hw * rw) / t.schur;
    const float step = part == 3 ? p : t.inverse * (r - component(t.ek, part + 1) * p);
    value = component(xi, part) + omega * step;
  }
  if (owner) reinterpret_cast<float*>(out)[threadIdx.x] = value;
  __syncthreads();
}

// A level's vectors: two iterates and the right-hand side, n each, from `at`.
// Sweeps start in the first iterate (from zero) or in `from`; the result's
// index, 0 or 1, is returned.
__device__ __forceinline__ int tail_smooth(int n, const TailHeld& t, float4* at, int from,
                                           int sweeps, bool zero, float omega, float4* staged) {
  for (int s = 0; s < sweeps; ++s) {
    const bool first = zero && s == 0;
    const int to = first ? 0 : from ^ 1;
    tail_pass(n, t, at + from * n, at + 2 * n, at + to * n, true, first, omega, staged);
    from = to;
  }
  return from;
}

__global__ void __launch_bounds__(kTailThreads) k_cpl_tail(const CoupledTail t) {
  extern __shared__ float4 tail_shared[];
  float4* staged = tail_shared;
  float4* vectors = tail_shared + CoupledTail::kMaxEntries;
  TailHeld held;
  tail_hold(t.op[0], held);
  pdl_entry();
  const int last = t.levels - 1;
  // The iterate of a level after its pre-sweeps, then after its post-sweeps.
  const int down = (t.pre - 1) & 1, up = (down + t.post) & 1;
  float4* v = vectors;
  for (int i = threadIdx.x; i < t.op[0].n; i += kTailThreads) v[2 * t.op[0].n + i] = t.b[i];
  __syncthreads();
  for (int k = 0; k < last; ++k) {
    const int n = t.op[k].n, below = t.op[k + 1].n;
    if (k > 0) tail_hold(t.op[k], held);
    tail_smooth(n, held, v, 0, t.pre, true, t.omega, staged);
    float4* r = v + (down ^ 1) * n;
    tail_pass(n, held, v + down * n, v + 2 * n, r, false, false, t.omega, staged);
    const CoupledTransfer& tr = t.down[k];
    float4* next = v + 3 * n;
    for (int at = threadIdx.x; at < 4 * below; at += kTailThreads) {
      const int i = at >> 2, part = at & 3;
      float s = 0.0f;
      const int end = tr.offsets[i + 1];
#pragma unroll 4
      for (int m = tr.offsets[i]; m < end; ++m)
        s += reinterpret_cast<const float*>(r)[4 * tr.members[m] + part];
      reinterpret_cast<float*>(next + 2 * below)[at] = s;
    }
    __syncthreads();
    v = next;
  }
  if (last > 0) tail_hold(t.op[last], held);
  int ends = tail_smooth(t.op[last].n, held, v, 0, t.coarsest, true, t.omega, staged);
  for (int k = last - 1; k >= 0; --k) {
    const float4* correction = v + ends * t.op[k + 1].n;
    const int n = t.op[k].n;
    v -= 3 * n;
    tail_hold(t.op[k], held);
    for (int i = threadIdx.x; i < n; i += kTailThreads)
      v[down * n + i] = plus(v[down * n + i], correction[t.down[k].aggregate[i]]);
    __syncthreads();
    tail_smooth(n, held, v, down, t.post, false, t.omega, staged);
    ends = up;
  }
  for (int i = threadIdx.x; i < t.op[0].n; i += kTailThreads) t.x[i] = v[ends * t.op[0].n + i];
}

int blocks_of(int items, int per) { return (items + per - 1) / per; }

// 32 rows and 512 staged entries per block of 128 threads where the rows fill
// the machine (110,842 rows of 12.6 entries: 14.7 us a sweep against 16.0 with 16
// rows and 23.7 with 256 threads; 24,652: 3.3, 4.7 and 6.4), 16 rows where more
// blocks shorten the sweep (14,318 rows of 15.6: 3.7 us against 4.6; 2,147: 3.1
// against 3.8; 423: 2.1 against 2.6). A thread per row took 17 to 24 us, 7.6, 7.2
// and 6.3 us on these levels.
constexpr int kWideRows = 1 << 14;
template <Pass kPass>
void coarse_rows(const CoupledLevel& l, const float4* x, const float4* b, float4* out, float omega,
                 const int* aggregate, const float4* coarse, cudaStream_t s) {
  if (l.n > kWideRows)
    pdl(k_cpl_coarse_rows<128, 32, 4, kPass>, blocks_of(l.n, 32), 128, 0, s, l, x, b, out, omega,
        aggregate, coarse);
  else
    pdl(k_cpl_coarse_rows<128, 16, 2, kPass>, blocks_of(l.n, 16), 128, 0, s, l, x, b, out, omega,
        aggregate, coarse);
}

}  // namespace

namespace launch {

template <class Term>
void cpl_terms_fine(const CoupledLevel& l, const CoupledTransfer& t, const CoupledMeshDevice& m,
                    int* count, Term* terms, int* term_faces, cudaStream_t s) {
  if (l.n <= 0) return;
  ++counter;
  k_cpl_terms_fine<Term><<<blocks_of(l.n, kBlock), kBlock, 0, s>>>(
      l, t, m.n, m.offsets, m.adjacent, m.faces, count, terms, term_faces);
}

template <class Term>
void cpl_terms_coarse(const CoupledLevel& l, const CoupledTransfer& t, const CoupledLevel& f,
                      int* count, Term* terms, cudaStream_t s) {
  if (l.n <= 0) return;
  ++counter;
  k_cpl_terms_coarse<Term><<<blocks_of(l.n, kBlock), kBlock, 0, s>>>(l, t, f, count, terms);
}

template void cpl_terms_fine<int>(const CoupledLevel&, const CoupledTransfer&,
                                  const CoupledMeshDevice&, int*, int*, int*, cudaStream_t);
template void cpl_terms_fine<long long>(const CoupledLevel&, const CoupledTransfer&,
                                        const CoupledMeshDevice&, int*, long long*, int*,
                                        cudaStream_t);
template void cpl_terms_coarse<int>(const CoupledLevel&, const CoupledTransfer&,
                                    const CoupledLevel&, int*, int*, cudaStream_t);
template void cpl_terms_coarse<long long>(const CoupledLevel&, const CoupledTransfer&,
                                          const CoupledLevel&, int*, long long*, cudaStream_t);

void cpl_galerkin_fine(const CoupledLevel& l, const CoupledFine& op, const float* cell, int cells,
                       float wc, cudaStream_t s) {
  const std::size_t n = static_cast<std::size_t>(cells);
  if (l.long_terms != nullptr)
    galerkin(l, FromFine<long long>{op, l.long_terms, l.term_faces, cell, n, wc}, s);
  else
    galerkin(l, FromFine<int>{op, l.terms, l.term_faces, cell, n, wc}, s);
}

void cpl_galerkin_coarse(const CoupledLevel& l, const CoupledLevel& f, cudaStream_t s) {
  if (l.long_terms != nullptr)
    galerkin(l, FromLevel<long long>{f, l.long_terms}, s);
  else
    galerkin(l, FromLevel<int>{f, l.terms}, s);
}

void cpl_coarse_prepare(const CoupledLevel& l, float* scratch, cudaStream_t s) {
  if (l.n <= 0) return;
  counter += 2;
  pdl(k_cpl_coarse_gsum, blocks_of(4 * l.n, kBlock), kBlock, 0, s, l, scratch);
  pdl(k_cpl_coarse_schur, blocks_of(8 * l.n, kBlock), kBlock, 0, s, l,
      static_cast<const float*>(scratch));
}

void cpl_coarse_residual(const CoupledLevel& l, const float4* x, const float4* b, float4* r,
                         cudaStream_t s) {
  if (l.n <= 0) return;
  ++counter;
  coarse_rows<Pass::Residual>(l, x, b, r, 0.0f, nullptr, nullptr, s);
}

void cpl_coarse_smooth(const CoupledLevel& l, const float4* x, const float4* b, float4* next,
                       float omega, bool first, const int* aggregate, const float4* coarse,
                       cudaStream_t s) {
  if (l.n <= 0) return;
  ++counter;
  if (first)
    pdl(k_cpl_coarse_first, blocks_of(4 * l.n, kBlock), kBlock, 0, s, l, b, next, omega);
  else if (aggregate != nullptr)
    coarse_rows<Pass::SmoothProlonged>(l, x, b, next, omega, aggregate, coarse, s);
  else
    coarse_rows<Pass::Smooth>(l, x, b, next, omega, nullptr, nullptr, s);
}

void cpl_restrict(int nc, const int* offsets, const int* members, const float4* fine,
                  float4* coarse, const CoupledLevel* l, float omega, float4* next,
                  cudaStream_t s) {
  if (nc <= 0) return;
  ++counter;
  if (next != nullptr)
    pdl(k_cpl_restrict<true>, blocks_of(4 * nc, kBlock), kBlock, 0, s, nc, offsets, members, fine,
        coarse, *l, omega, next);
  else
    pdl(k_cpl_restrict<false>, blocks_of(4 * nc, kBlock), kBlock, 0, s, nc, offsets, members, fine,
        coarse, CoupledLevel{}, omega, next);
}

void cpl_tail(const CoupledTail& t, cudaStream_t s) {
  if (t.levels <= 0) return;
  ++counter;
  int rows = 0;
  for (int k = 0; k < t.levels; ++k) rows += t.op[k].n;
  const auto bytes = [](int all) {
    return (CoupledTail::kMaxEntries + 3 * all) * static_cast<int>(sizeof(float4));
  };
  static std::atomic<unsigned long long> raised{0};
  raise_shared_limit(reinterpret_cast<const void*>(k_cpl_tail),
                     bytes(CoupledTail::kMaxLevels * CoupledTail::kMaxRows), raised);
  pdl(k_cpl_tail, 1, kTailThreads, bytes(rows), s, t);
}

}  // namespace launch
}  // namespace kb2
