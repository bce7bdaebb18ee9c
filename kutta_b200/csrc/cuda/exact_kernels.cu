// Reference-parity solver kernels for sm_100a (compiled with --fmad=false).
//
// Each kernel computes exactly the float operations, in exactly the order, of
// the reference kernel it replaces (cited per kernel), so every per-row value is
// bit-identical to the reference's CPU path. Reductions accumulate in FP64 in a
// fixed tree; they are fused into the kernel that produces their operand and the
// last block runs the reference's single-thread scalar update as an epilogue,
// so a PCG iteration is a handful of launches instead of a dozen.
#include "bf16_rows.cuh"
#include "common.cuh"
#include "epilogues.cuh"
#include "kernels.hpp"

#include <algorithm>
#include <atomic>
#include <cstdlib>

namespace kb2 {
namespace dev {
bool pdl_enabled() {
  static const bool enabled = [] {
    const char* v = std::getenv("KUTTA_B200_PDL");
    return v == nullptr || v[0] != '0';
  }();
  return enabled;
}
}  // namespace dev
namespace {
using namespace dev;

#define ROWS(i, n) \
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

// ---- CSR row kernels --------------------------------------------------------
// One row per thread: on the 5-entry fine rows this direct form measured
// fastest; staging tiles in shared memory or
// register-chunking the row both measured slower there.

// The column of entry j of row i: from the CSR columns, or with kNear from 16-bit
// offsets from the row (a level whose columns all lie that near). These kernels
// are bound by HBM, and an entry is then 6 bytes instead of 8: a sweep over
// 2,097,152 rows of seven entries 26.3 us instead of 28.3, over 1,572,864 rows of
// five 15.3 instead of 18.5.
template <bool kNear>
struct Columns {
  const void* data;
  __device__ __forceinline__ int operator()(int i, int j) const {
    if constexpr (kNear) return i + __ldg(static_cast<const short*>(data) + j);
    return __ldg(static_cast<const int*>(data) + j);
  }
};
__global__ void k_near_offsets(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                               short* __restrict__ near) {
  pdl_entry();
  ROWS(i, n) for (int j = rows[i]; j < rows[i + 1]; ++j) near[j] = static_cast<short>(cols[j] - i);
}

// csr_spmv / csr_spmv_guarded, linalg.kern.h:5-16,111-114.
__global__ void k_spmv(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                       const float* __restrict__ vals, const float* __restrict__ x,
                       float* __restrict__ y, const int* __restrict__ status) {
  pdl_entry();
  if (status && status[0] != 0) return;
  ROWS(i, n) {
    float sum = 0.0f, error = 0.0f;
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) kahan_term(sum, error, vals[j], x[cols[j]]);
    y[i] = sum;
  }
}

// csr_spmv_guarded + dot_into(w, q) + a scalar kernel: PCG's p.q and alpha
// (solver.cpp:288-290, w = p) or BiCGStab's rhat.q and alpha (:335-337, w = rhat).
template <bool kNear>
__global__ void k_spmv_dot(int n, const int* __restrict__ rows, Columns<kNear> cols,
                           const float* __restrict__ vals, const float* __restrict__ p,
                           const float* __restrict__ w, float* __restrict__ q, DeviceReducer red,
                           float* scalars, int offset, int* status, Epilogue epi) {
  pdl_entry();
  if (status[0] != 0) return;
  double acc = 0;
  ROWS(i, n) {
    float sum = 0.0f, error = 0.0f;
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) kahan_term(sum, error, vals[j], p[cols(i, j)]);
    q[i] = sum;
    acc += static_cast<double>(w[i]) * static_cast<double>(sum);
  }
  finish(as_reducer(red), acc, 0, false, scalars, offset, status, epi);
}

// csr_spmv_guarded + dot2_into(t, t; t, s) + solver_bicg_omega (solver.cpp:343-347).
template <bool kNear>
__global__ void k_spmv_dot2(int n, const int* __restrict__ rows, Columns<kNear> cols,
                            const float* __restrict__ vals, const float* __restrict__ x,
                            const float* __restrict__ sv, float* __restrict__ t, DeviceReducer red,
                            float* scalars, int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  double tt = 0, ts = 0;
  ROWS(i, n) {
    float sum = 0.0f, error = 0.0f;
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) kahan_term(sum, error, vals[j], x[cols(i, j)]);
    t[i] = sum;
    tt += static_cast<double>(sum) * static_cast<double>(sum);
    ts += static_cast<double>(sum) * static_cast<double>(sv[i]);
  }
  finish(as_reducer(red), tt, ts, true, scalars, 2, status, Epilogue::BicgOmega);
}

// csr_residual / csr_residual_guarded, linalg.kern.h:32-50,115-118.
template <bool kNear>
__global__ void k_residual(int n, const int* __restrict__ rows, Columns<kNear> cols,
                           const float* __restrict__ vals, const float* __restrict__ x,
                           const float* __restrict__ b, float* __restrict__ r,
                           const int* __restrict__ status) {
  pdl_entry();
  if (status && status[0] != 0) return;
  ROWS(i, n) {
    float sum = b[i], error = 0.0f;
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) residual_term(sum, error, vals[j], x[cols(i, j)]);
    r[i] = sum + error;
  }
}

// amg_smooth (linalg.kern.h:150-156) and amg_smooth_zero (:162-170).
template <bool kZero, bool kNear>
__global__ void k_smooth(int n, const int* __restrict__ rows, Columns<kNear> cols,
                         const float* __restrict__ vals, const float* __restrict__ x,
                         const float* __restrict__ b, const float* __restrict__ inv,
                         float* __restrict__ next, const int* __restrict__ status) {
  pdl_entry();
  if (status && status[0] != 0) return;
  ROWS(i, n) {
    if (kZero) {
      next[i] = zero_sweep_row(i, rows, vals, b[i], inv[i]);
      continue;
    }
    float sum = b[i], error = 0.0f;
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) residual_term(sum, error, vals[j], x[cols(i, j)]);
    next[i] = x[i] + (2.0f / 3.0f) * inv[i] * (sum + error);
  }
}

// The fine-level post-sweep of the flexible PCG (mixed solve) with the two
// reductions that follow the preconditioner fused in: next as
// k_smooth<false>, then b.next and next.q (b the Krylov residual r, next the
// preconditioned z, q = A p) into scalars[offset..] with the epilogue, as
// reduce_into(Dot2, r, z, z, q) computes them: the same grid, the same row
// loop and the same products, so the same totals bit for bit.
__global__ void k_smooth_dot2(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                              const float* __restrict__ vals, const float* __restrict__ x,
                              const float* __restrict__ b, const float* __restrict__ inv,
                              float* __restrict__ next, const float* __restrict__ q,
                              DeviceReducer red, float* scalars, int offset, int* status,
                              Epilogue epi) {
  pdl_entry();
  if (status[0] != 0) return;
  double a = 0, c = 0;
  ROWS(i, n) {
    float sum = b[i], error = 0.0f;
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) residual_term(sum, error, vals[j], x[cols[j]]);
    const float z = x[i] + (2.0f / 3.0f) * inv[i] * (sum + error);
    next[i] = z;
    a += static_cast<double>(b[i]) * static_cast<double>(z);
    c += static_cast<double>(z) * static_cast<double>(q[i]);
  }
  finish(as_reducer(red), a, c, true, scalars, offset, status, epi);
}

// ---- Packed rows (the mixed solve's fine operator) ---------------------------
// The kernels are bounded to 32 registers a thread (8 blocks of 256 per SM):
// their grids are the CSR kernels' (8 blocks per SM, one resident wave), and
// at more registers part of the grid would wait for a second wave.
// The row's values, absolute columns and diagonal, loaded with 128-bit (and
// 64-bit) loads that stream past the caches: the operator is read once per
// pass, the gathered vectors are what the caches should keep.
template <int W>
struct PackedRow {
  float v[W];
  int c[W];
  float d;
};
template <int W>
__device__ __forceinline__ PackedRow<W> packed_row(int i, const float* __restrict__ vals,
                                                   const short* __restrict__ offsets,
                                                   const float* __restrict__ diag) {
  PackedRow<W> row;
  const float4* v4 = reinterpret_cast<const float4*>(vals) + static_cast<std::size_t>(i) * (W / 4);
#pragma unroll
  for (int q = 0; q < W / 4; ++q) {
    const float4 a = __ldcs(v4 + q);
    row.v[4 * q] = a.x;
    row.v[4 * q + 1] = a.y;
    row.v[4 * q + 2] = a.z;
    row.v[4 * q + 3] = a.w;
  }
  unsigned words[W / 2];
  if constexpr (W == 4) {
    const uint2 o = __ldcs(reinterpret_cast<const uint2*>(offsets) + i);
    words[0] = o.x;
    words[1] = o.y;
  } else {
    const uint4 o = __ldcs(reinterpret_cast<const uint4*>(offsets) + i);
    words[0] = o.x;
    words[1] = o.y;
    words[2] = o.z;
    words[3] = o.w;
  }
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const int off = static_cast<short>((words[k / 2] >> (16 * (k & 1))) & 0xffffu);
    row.c[k] = i + off;
  }
  row.d = __ldcs(diag + i);
  return row;
}

// residual_term with the product's rounding error taken by one FMA instead of
// Dekker's 4097 split: both give the exact error of v x when neither factor
// exceeds 1e30 (the split's guard, kept) and no partial product underflows,
// so the sums agree bit for bit there at a third of the instructions, which
// keeps these streaming kernels memory-bound.
__device__ __forceinline__ void residual_term_fma(float& sum, float& error, float v, float x) {
  const float product = v * x;
  const float term = -product;
  const float next = sum + term;
  error += fabsf(sum) >= fabsf(term) ? (sum - next) + term : (term - next) + sum;
  if (fabsf(v) <= 1.0e30f && fabsf(x) <= 1.0e30f) error -= fmaf(v, x, -product);
  sum = next;
}

// sum = b_i - sum_j a_ij x_j with residual_term_fma, in CSR column order;
// unused slots (column i) are skipped.
template <int W>
__device__ __forceinline__ float packed_residual_row(int i, const PackedRow<W>& row, float bi,
                                                     const float* __restrict__ x) {
  float xv[W];
#pragma unroll
  for (int k = 0; k < W; ++k) xv[k] = x[row.c[k]];
  const float xi = x[i];
  float sum = bi, error = 0.0f;
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (row.c[k] < i) residual_term_fma(sum, error, row.v[k], xv[k]);
  residual_term_fma(sum, error, row.d, xi);
#pragma unroll
  for (int k = 0; k < W; ++k)
    if (row.c[k] > i) residual_term_fma(sum, error, row.v[k], xv[k]);
  return sum + error;
}

template <int W>
__global__ void __launch_bounds__(kBlock, 8) k_packed_residual(int n, const float* __restrict__ vals,
                                  const short* __restrict__ offsets, const float* __restrict__ diag,
                                  const float* __restrict__ x, const float* __restrict__ b,
                                  float* __restrict__ r, const int* __restrict__ status) {
  pdl_entry();
  if (status && status[0] != 0) return;
  ROWS(i, n) {
    const PackedRow<W> row = packed_row<W>(i, vals, offsets, diag);
    r[i] = packed_residual_row<W>(i, row, b[i], x);
  }
}

// k_smooth_dot2 on packed rows.
template <int W>
__global__ void __launch_bounds__(kBlock, 8) k_packed_smooth_dot2(int n, const float* __restrict__ vals,
                                     const short* __restrict__ offsets,
                                     const float* __restrict__ diag, const float* __restrict__ x,
                                     const float* __restrict__ b, const float* __restrict__ inv,
                                     float* __restrict__ next, const float* __restrict__ q,
                                     DeviceReducer red, float* scalars, int offset, int* status,
                                     Epilogue epi) {
  pdl_entry();
  if (status[0] != 0) return;
  double a = 0, c = 0;
  ROWS(i, n) {
    const PackedRow<W> row = packed_row<W>(i, vals, offsets, diag);
    const float bi = b[i];
    const float z = x[i] + (2.0f / 3.0f) * inv[i] * packed_residual_row<W>(i, row, bi, x);
    next[i] = z;
    a += static_cast<double>(bi) * static_cast<double>(z);
    c += static_cast<double>(z) * static_cast<double>(q[i]);
  }
  finish(as_reducer(red), a, c, true, scalars, offset, status, epi);
}

// k_spmv_dot on packed rows (Kahan sum in CSR column order).
template <int W>
__global__ void __launch_bounds__(kBlock, 8) k_packed_spmv_dot(int n, const float* __restrict__ vals,
                                  const short* __restrict__ offsets,
                                  const float* __restrict__ diag, const float* __restrict__ p,
                                  const float* __restrict__ w, float* __restrict__ q,
                                  DeviceReducer red, float* scalars, int offset, int* status,
                                  Epilogue epi) {
  pdl_entry();
  if (status[0] != 0) return;
  double acc = 0;
  ROWS(i, n) {
    const PackedRow<W> row = packed_row<W>(i, vals, offsets, diag);
    float pv[W];
#pragma unroll
    for (int k = 0; k < W; ++k) pv[k] = p[row.c[k]];
    const float pi = p[i];
    float sum = 0.0f, error = 0.0f;
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (row.c[k] < i) kahan_term(sum, error, row.v[k], pv[k]);
    kahan_term(sum, error, row.d, pi);
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (row.c[k] > i) kahan_term(sum, error, row.v[k], pv[k]);
    q[i] = sum;
    acc += static_cast<double>(w[i]) * static_cast<double>(sum);
  }
  finish(as_reducer(red), acc, 0, false, scalars, offset, status, epi);
}

// Values of the packed rows: the row's off-diagonal values in column order,
// then zeros; the diagonal apart.
__global__ void k_pack_rows(int n, int width, const int* __restrict__ rows,
                            const int* __restrict__ diag_index, const float* __restrict__ vals,
                            float* __restrict__ packed, float* __restrict__ packed_diag) {
  pdl_entry();
  ROWS(i, n) pack_row(i, width, rows, diag_index, vals, packed, packed_diag);
}

// amg_coarse_solve, linalg.kern.h:126-147: the whole <=24-row system in one
// warp, a lane per row. Each lane sums its row in CSR order and the iterate is
// exchanged through shared memory, so every value is the one-thread form's;
// the operator is read once into shared memory. 32 sweeps of 8 rows took
// 67 us in one thread (each entry a dependent load).
__global__ void k_coarse_solve(int count, const int* __restrict__ rows,
                               const int* __restrict__ cols, const float* __restrict__ vals,
                               float* __restrict__ x, const float* __restrict__ b,
                               const float* __restrict__ inv, const int* __restrict__ status,
                               int sweeps) {
  pdl_entry();
  if (status[0] != 0) return;
  constexpr int kMost = 24;
  __shared__ float current[kMost];
  __shared__ int col[kMost * kMost];
  __shared__ float val[kMost * kMost];
  const int row = threadIdx.x;
  const bool owner = row < count;
  const int nnz = rows[count];
  for (int j = row; j < nnz; j += 32) {
    col[j] = cols[j];
    val[j] = vals[j];
  }
  if (owner) current[row] = 0.0f;
  const int begin = owner ? rows[row] : 0, end = owner ? rows[row + 1] : 0;
  const float right = owner ? b[row] : 0.0f, scale = owner ? inv[row] : 0.0f;
  __syncwarp();
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    float sum = right, error = 0.0f;
#pragma unroll 4
    for (int j = begin; j < end; ++j) residual_term(sum, error, val[j], current[col[j]]);
    const float r = sum + error;
    __syncwarp();
    if (owner) current[row] += (2.0f / 3.0f) * scale * r;
    __syncwarp();
  }
  if (owner) x[row] = current[row];
}

// krylov_diagonal, linalg.kern.h:52-70, with the refresh's max_abs check of the
// invalid flags fused (amg.cpp:236-240).
__global__ void k_diagonal(int n, const int* __restrict__ rows, const int* __restrict__ diag,
                           const float* __restrict__ vals, float* __restrict__ inverse,
                           int use_l1, DeviceReducer red, double* check, int slot) {
  pdl_entry();
  double worst = 0;
  ROWS(i, n) worst = nan_max(worst, diagonal_row<false>(i, rows, diag, vals, inverse, use_l1));
  finish_max(as_reducer(red), worst, check, slot);
}

// ---- AMG transfer and Galerkin, src/kutta/kernels/amg.kern.h ------------------
// amg_prolong(_guarded) :18-21,88-91.
__global__ void k_prolong(int nf, const int* __restrict__ aggregate,
                          const float* __restrict__ coarse, float* __restrict__ fine,
                          const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  ROWS(i, nf) {
    const int g = aggregate[i];
    if (g >= 0) fine[i] += coarse[g];
  }
}

// amg_galerkin :27-38: Neumaier sum over the coarse entry's fine entries. An
// off-diagonal entry has one to a few of them, a diagonal some thirty, and a
// warp walks as far as its longest list; so the diagonals, marked in `diagonal`
// (a bit per entry), are summed by blocks of their own, a thread per row
// (Diagonals::Apart), or not at all where the M-matrix diagonal replaces them
// (Diagonals::Left). Levels of at most kApartEntries take all entries alike
// (Diagonals::Along): 86,950 entries 4.3 us against 5.2, 251,223 6.5 against 5.3.
enum class Diagonals { Left, Apart, Along };
constexpr int kApartEntries = 1 << 17;
template <Diagonals kDiagonals>
__global__ void k_galerkin(int n_c, int nnz_c, const int* __restrict__ offsets,
                           const int* __restrict__ entries, const unsigned* __restrict__ diagonal,
                           const int* __restrict__ diag, const float* __restrict__ fine,
                           float* __restrict__ coarse, int diagonal_blocks) {
  pdl_entry();
  const auto sum_list = [&](int e) {
    float sum = 0.0f, error = 0.0f;
    const int end = offsets[e + 1];
    for (int j = offsets[e]; j < end; ++j) neumaier_term(sum, error, fine[entries[j]]);
    coarse[e] = sum + error;
  };
  const int block = static_cast<int>(blockIdx.x) - diagonal_blocks;
  if (kDiagonals == Diagonals::Apart && block < 0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_c) sum_list(diag[i]);
    return;
  }
  const int stride = (gridDim.x - diagonal_blocks) * blockDim.x;
  for (int e = block * blockDim.x + threadIdx.x; e < nnz_c; e += stride)
    if (kDiagonals == Diagonals::Along || !(diagonal[e >> 5] >> (e & 31) & 1u)) sum_list(e);
}

// The bits of the diagonal entries (words zeroed before).
__global__ void k_mark_diagonals(int n, const int* __restrict__ diag,
                                 unsigned* __restrict__ words) {
  pdl_entry();
  ROWS(i, n) atomicOr(words + (diag[i] >> 5), 1u << (diag[i] & 31));
}

// amg_m_matrix_diagonal :44-58 in two passes with the same roundings in the
// same order: each fine row's surplus (its diagonal plus its off-diagonals,
// upward rounded), independent per row and computed in parallel; then, per
// coarse row, the upward-rounded sum of its members' surpluses in member
// order minus its stored off-diagonals. Splitting the member loop out of the
// per-coarse-row chain shortens the dependent sequence of each thread.
__global__ void k_row_surplus(int n, const int* __restrict__ rows, const int* __restrict__ diag,
                              const float* __restrict__ fine, float* __restrict__ surplus) {
  pdl_entry();
  ROWS(i, n) surplus[i] = row_surplus(i, rows, diag, fine);
}

__global__ void k_m_matrix_combine(int nc, const int* __restrict__ offsets,
                                   const int* __restrict__ members,
                                   const float* __restrict__ surplus, const int* __restrict__ rows,
                                   const int* __restrict__ diag, float* coarse) {
  pdl_entry();
  ROWS(g, nc) {
    UpperSum diagonal{0.0f, 0.0f};
    for (int m = offsets[g]; m < offsets[g + 1]; ++m)
      diagonal = upper_add(diagonal, surplus[members[m]]);
    for (int j = rows[g]; j < rows[g + 1]; ++j)
      if (j != diag[g]) diagonal = upper_add(diagonal, -coarse[j]);
    coarse[diag[g]] = upper_value(diagonal);
  }
}

// A level's row data in one pass of a refresh, where each was a launch of its
// own: with kCombine the M-matrix diagonal (k_m_matrix_combine), then the
// inverse L1 diagonal and its invalid flag (k_diagonal), and where wanted the
// row's surplus for the level below (k_row_surplus) and its BF16 copy
// (k_bf16_pack). A thread's row stays in L1 between the parts, and every part
// is the same operations in the same order. (Staging a block's rows in shared
// memory was slower: the upward-rounded chains bound it, not the loads; eight
// loads in flight took the levels of a 1.57M-row tet hierarchy from 101 to 96 us.)
template <bool kCombine>
__global__ void k_level_rows(int n, const int* __restrict__ rows, const int* __restrict__ diag,
                             float* vals, const int* __restrict__ offsets,
                             const int* __restrict__ members,
                             const float* __restrict__ fine_surplus, float* __restrict__ inverse,
                             float* __restrict__ surplus, Bf16Store store, DeviceReducer red,
                             double* check, int slot) {
  pdl_entry();
  double worst = 0;
  ROWS(i, n) {
    if constexpr (kCombine) {
      constexpr int kBatch = 8;
      UpperSum diagonal{0.0f, 0.0f};
      const int end = offsets[i + 1];
      for (int m = offsets[i]; m < end; m += kBatch) {
        float v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) v[k] = m + k < end ? fine_surplus[members[m + k]] : 0.0f;
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
          if (m + k < end) diagonal = upper_add(diagonal, v[k]);
      }
      const int at = diag[i];
      row_values(vals, rows[i], rows[i + 1], [&](int j, float v) {
        if (j != at) diagonal = upper_add(diagonal, -v);
      });
      vals[at] = upper_value(diagonal);
    }
    worst = nan_max(worst, diagonal_row(i, rows, diag, vals, inverse, 1));
    if (surplus != nullptr) surplus[i] = row_surplus(i, rows, diag, vals);
    if (store.scale != nullptr) bf16_store_row(i, vals, store);
  }
  finish_max(as_reducer(red), worst, check, slot);
}

// ---- Krylov vector updates, scalars.kern.h:122-152 ---------------------------
// solver_step :122-127 + dot_into(r, r -> 18) + solver_check(pcg) (solver.cpp:291-293);
// with next != null also the fine level's zero-start sweep of the new r, which
// the AMG cycle begins with (it reads r and writes the sweep: 4 of its 12 bytes a
// row and a launch less).
__global__ void k_pcg_step_dot(int n, float* __restrict__ x, float* __restrict__ r,
                               const float* __restrict__ p, const float* __restrict__ q,
                               const int* __restrict__ rows, const float* __restrict__ vals,
                               const float* __restrict__ inv, float* __restrict__ next,
                               DeviceReducer red, float* scalars, int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  const float alpha = kp_float(kp_load(scalars, 8));
  double acc = 0;
  ROWS(i, n) {
    x[i] += alpha * p[i];
    const float ri = r[i] - alpha * q[i];
    r[i] = ri;
    if (next != nullptr) next[i] = zero_sweep_row(i, rows, vals, ri, inv[i]);
    acc += static_cast<double>(ri) * static_cast<double>(ri);
  }
  finish(as_reducer(red), acc, 0, false, scalars, 18, status, Epilogue::CheckPcg);
}

// solver_direction :128-131.
__global__ void k_direction(int n, const float* __restrict__ z, float* __restrict__ p,
                            const float* __restrict__ scalars, const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  const float beta = kp_float(kp_load(scalars, 10));
  ROWS(i, n) p[i] = z[i] + beta * p[i];
}

// solver_bicg_direction :132-137.
__global__ void k_bicg_direction(int n, const float* __restrict__ r, const float* __restrict__ v,
                                 float* __restrict__ p, const float* __restrict__ scalars,
                                 const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  const float beta = kp_float(kp_load(scalars, 10)), omega = kp_float(kp_load(scalars, 12));
  ROWS(i, n) p[i] = r[i] + beta * (p[i] - omega * v[i]);
}

// solver_bicg_difference :138-141 + dot_into(s, s -> 16) + solver_bicg_s.
__global__ void k_bicg_difference(int n, const float* __restrict__ r, const float* __restrict__ q,
                                  float* __restrict__ sv, DeviceReducer red, float* scalars,
                                  int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  const float alpha = kp_float(kp_load(scalars, 8));
  double acc = 0;
  ROWS(i, n) {
    const float si = r[i] - alpha * q[i];
    sv[i] = si;
    acc += static_cast<double>(si) * static_cast<double>(si);
  }
  finish(as_reducer(red), acc, 0, false, scalars, 16, status, Epilogue::BicgS);
}

// solver_bicg_step :142-149 + dot_into(r, r -> 18) + solver_check, and the next
// update's dot_into(rhat, r -> 0) + solver_bicg_beta.
__global__ void k_bicg_step(int n, float* __restrict__ x, float* __restrict__ r,
                            const float* __restrict__ z, const float* __restrict__ zs,
                            const float* __restrict__ sv, const float* __restrict__ t,
                            const float* __restrict__ shadow, DeviceReducer red, float* scalars,
                            int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  const float alpha = kp_float(kp_load(scalars, 8)), omega = kp_float(kp_load(scalars, 12));
  const bool s_only = status[2] != 0;
  double rr = 0, rho = 0;
  ROWS(i, n) {
    float ri;
    if (s_only) {
      x[i] += alpha * z[i];
      ri = sv[i];
    } else {
      x[i] += alpha * z[i] + omega * zs[i];
      ri = sv[i] - omega * t[i];
    }
    r[i] = ri;
    rr += static_cast<double>(ri) * static_cast<double>(ri);
    rho += static_cast<double>(shadow[i]) * static_cast<double>(ri);
  }
  finish_bicg(as_reducer(red), rr, rho, scalars, status);
}

// krylov_multiply(_guarded), linalg.kern.h:72-75,119-122.
__global__ void k_multiply(int n, const float* __restrict__ r, const float* __restrict__ inverse,
                           float* __restrict__ z, const int* __restrict__ status) {
  pdl_entry();
  if (status && status[0] != 0) return;
  ROWS(i, n) z[i] = r[i] * inverse[i];
}

// axpy, blas.kern.h:5.
__global__ void k_axpy(int n, float* __restrict__ y, const float* __restrict__ x, float a) {
  pdl_entry();
  ROWS(i, n) y[i] = y[i] + a * x[i];
}

__global__ void k_fill(int n, float* __restrict__ x, float value) {
  pdl_entry(); ROWS(i, n) x[i] = value; }

// ---- reductions ---------------------------------------------------------------
// Device::reduce_into (device.hpp:186-202) with FP64 accumulation.
__global__ void k_reduce_into(ReduceMode mode, int n, const float* __restrict__ x,
                              const float* __restrict__ y, const float* __restrict__ u,
                              const float* __restrict__ v, DeviceReducer red, float* scalars,
                              int offset, int* status, bool guard, Epilogue epi) {
  pdl_entry();
  if (guard && status[0] != 0) return;
  double a = 0, b = 0;
  const bool dual = mode == ReduceMode::Dot2;
  ROWS(i, n) {
    a += mode == ReduceMode::Sum ? static_cast<double>(x[i])
                                 : static_cast<double>(x[i]) * static_cast<double>(y[i]);
    if (dual) b += static_cast<double>(u[i]) * static_cast<double>(v[i]);
  }
  finish(as_reducer(red), a, b, dual, scalars, offset, status, epi);
}

// Host reductions (Device::sum/dot/max_abs): the FP64 value into out[slot].
__global__ void k_reduce_value(ReduceMode mode, int n, const float* __restrict__ x,
                               const float* __restrict__ y, DeviceReducer red, double* out,
                               int slot) {
  pdl_entry();
  __shared__ double shared[32];
  double a = 0;
  ROWS(i, n) {
    if (mode == ReduceMode::MaxAbs) a = nan_max(a, fabs(static_cast<double>(x[i])));
    else if (mode == ReduceMode::Sum) a += static_cast<double>(x[i]);
    else a += static_cast<double>(x[i]) * static_cast<double>(y[i]);
  }
  const Reducer r = as_reducer(red);
  a = mode == ReduceMode::MaxAbs ? block_max(a, shared) : block_sum(a, shared);
  if (!publish(r, a, 0, false)) return;
  const double total = mode == ReduceMode::MaxAbs ? gather_max(r, shared) : gather(r, 0, shared);
  if (threadIdx.x == 0) {
    out[slot] = total;
    *r.ticket = 0;
  }
}

// solver_limits :51-55 (all 24 slots).
__global__ void k_solver_limits(float* scalars, float th, float tl, float dh, float dl) {
  pdl_entry();
  const int i = threadIdx.x;
  if (i < 24)
    scalars[i] = i == 20 ? th : (i == 21 ? tl : (i == 22 ? dh : (i == 23 ? dl : 0.0f)));
}

// solver_reset :56-62.
__global__ void k_solver_reset(float* scalars, int* status, int iterations) {
  pdl_entry();
  status[0] = 0;
  status[1] = iterations;
  status[2] = 0;
  scalars[8] = 1.0f;
  scalars[9] = 0.0f;
  scalars[12] = 1.0f;
  scalars[13] = 0.0f;
  scalars[14] = 1.0f;
  scalars[15] = 0.0f;
}

// solver_project :150-152.
__global__ void k_project(int n, float* __restrict__ x, const float* __restrict__ sum,
                          float count_hi, float count_lo) {
  pdl_entry();
  const float mean = kp_float(kp_div(kp_load(sum, 0), kp(count_hi, count_lo)));
  ROWS(i, n) x[i] -= mean;
}

// ---- K-cycle inner corrections (scalars.kern.h:154-186) ------------------------
// Per-level scalars: [0] p.q (q.q for GCR), [2] b.p / t.p (b.q / t.q), [4] t.t or
// z.q, [6] b.b, [8] alpha, [10] beta. The level's status: 0 running, 1 keep the
// accepted first correction, 2 fall back to the plain first cycle.
__global__ void k_inner_alpha(float* scalars, int* status, const int* parent, int first) {
  pdl_entry();
  if (first != 0) status[0] = parent[0] == 0 ? 0 : 2;
  if (status[0] != 0) return;
  const Pair denom = kp_load(scalars, 0);
  const Pair alpha = kp_div(kp_load(scalars, 2), denom);
  if (!kp_positive(denom) || !kp_coefficient(alpha) ||
      (kp_zero(alpha) && !kp_zero(kp_load(scalars, 2))))
    status[0] = first != 0 ? 2 : 1;
  else
    kp_store(scalars, 8, alpha);
}

__global__ void k_inner_first(int n, const float* __restrict__ b, const float* __restrict__ p,
                              const float* __restrict__ q, float* __restrict__ x,
                              float* __restrict__ t, const float* __restrict__ scalars,
                              const int* __restrict__ status) {
  pdl_entry();
  const bool running = status[0] == 0;
  const float alpha = kp_float(kp_load(scalars, 8));
  ROWS(i, n) {
    x[i] = running ? alpha * p[i] : p[i];
    t[i] = running ? b[i] - alpha * q[i] : 0.0f;
  }
}

// Adaptive exit: keep the first correction when |t|^2 <= |b|^2 / 16.
__global__ void k_inner_check(const float* scalars, int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  if (kp_le(kp_load(scalars, 4), kp_mul(kp(0.0625f, 0.0f), kp_load(scalars, 6)))) status[0] = 1;
}

__global__ void k_inner_beta(float* scalars, int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  const Pair beta = kp_div(kp_neg(kp_load(scalars, 4)), kp_load(scalars, 0));
  if (!kp_coefficient(beta) || (kp_zero(beta) && !kp_zero(kp_load(scalars, 4))))
    status[0] = 1;
  else
    kp_store(scalars, 10, beta);
}

__global__ void k_inner_step(int n, float* __restrict__ x, const float* __restrict__ p,
                             const float* __restrict__ scalars, const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  const float alpha = kp_float(kp_load(scalars, 8));
  ROWS(i, n) x[i] += alpha * p[i];
}

inline int blocks(int n) { return grid_for(n); }
// Kernels without a reduction: one row per thread below ~2M rows, where that
// measured fastest; above, the 1184-block grid-stride form measured faster
// (fine-level sweep 65.9 us vs 72.1 us at 5.3M rows).
inline int full_grid(int n) {
  if (n >= (1 << 21)) return grid_for(n);
  return n > 0 ? (n + kBlock - 1) / kBlock : 1;
}
static_assert(kReducePartials == kPartials, "reduction scratch size");

}  // namespace

namespace launch {

std::atomic<long long> counter{0};

void spmv(int n, const int* rows, const int* cols, const float* vals, const float* x, float* y,
          const int* status, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_spmv, full_grid(n), kBlock, 0, s, n, rows, cols, vals, x, y, status);
}
void spmv_dot(int n, const int* rows, const int* cols, const short* near, const float* vals,
              const float* p, const float* w, float* q, DeviceReducer red, float* scalars,
              int offset, int* status, Epilogue epi, cudaStream_t s) {
  ++counter;
  if (near)
    pdl(k_spmv_dot<true>, blocks(n), kBlock, 0, s, n, rows, Columns<true>{near}, vals, p, w, q, red,
        scalars, offset, status, epi);
  else
    pdl(k_spmv_dot<false>, blocks(n), kBlock, 0, s, n, rows, Columns<false>{cols}, vals, p, w, q,
        red, scalars, offset, status, epi);
}
void spmv_dot2(int n, const int* rows, const int* cols, const short* near, const float* vals,
               const float* x, const float* sv, float* t, DeviceReducer red, float* scalars,
               int* status, cudaStream_t s) {
  ++counter;
  if (near)
    pdl(k_spmv_dot2<true>, blocks(n), kBlock, 0, s, n, rows, Columns<true>{near}, vals, x, sv, t,
        red, scalars, status);
  else
    pdl(k_spmv_dot2<false>, blocks(n), kBlock, 0, s, n, rows, Columns<false>{cols}, vals, x, sv, t,
        red, scalars, status);
}
void residual(int n, const int* rows, const int* cols, const short* near, const float* vals,
              const float* x, const float* b, float* r, const int* status, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  if (near)
    pdl(k_residual<true>, full_grid(n), kBlock, 0, s, n, rows, Columns<true>{near}, vals, x, b, r,
        status);
  else
    pdl(k_residual<false>, full_grid(n), kBlock, 0, s, n, rows, Columns<false>{cols}, vals, x, b, r,
        status);
}
void smooth(int n, const int* rows, const int* cols, const short* near, const float* vals,
            const float* x, const float* b, const float* inv, float* next, const int* status,
            bool zero_start, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  if (zero_start)
    pdl(k_smooth<true, false>, full_grid(n), kBlock, 0, s, n, rows, Columns<false>{cols}, vals, x, b,
        inv, next, status);
  else if (near)
    pdl(k_smooth<false, true>, full_grid(n), kBlock, 0, s, n, rows, Columns<true>{near}, vals, x, b,
        inv, next, status);
  else
    pdl(k_smooth<false, false>, full_grid(n), kBlock, 0, s, n, rows, Columns<false>{cols}, vals, x,
        b, inv, next, status);
}
void near_offsets(int n, const int* rows, const int* cols, short* near, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_near_offsets, full_grid(n), kBlock, 0, s, n, rows, cols, near);
}
void smooth_dot2(int n, const int* rows, const int* cols, const float* vals, const float* x,
                 const float* b, const float* inv, float* next, const float* q, DeviceReducer red,
                 float* scalars, int offset, int* status, Epilogue epi, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_smooth_dot2, blocks(n), kBlock, 0, s, n, rows, cols, vals, x, b, inv, next, q, red,
                                             scalars, offset, status, epi);
}
void pack_rows(int n, int width, const int* rows, const int* cols, const int* diag,
               const float* vals, float* packed, float* packed_diag, cudaStream_t s) {
  (void)cols;
  if (n <= 0) return;
  ++counter;
  pdl(k_pack_rows, full_grid(n), kBlock, 0, s, n, width, rows, diag, vals, packed, packed_diag);
}
void packed_residual(int n, PackedRows a, const float* x, const float* b, float* r,
                     const int* status, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  if (a.width == 4)
    pdl(k_packed_residual<4>, full_grid(n), kBlock, 0, s, n, a.vals, a.offsets, a.diag, x, b, r,
        status);
  else
    pdl(k_packed_residual<8>, full_grid(n), kBlock, 0, s, n, a.vals, a.offsets, a.diag, x, b, r,
        status);
}
void packed_spmv_dot(int n, PackedRows a, const float* p, const float* w, float* q,
                     DeviceReducer red, float* scalars, int offset, int* status, Epilogue epi,
                     cudaStream_t s) {
  ++counter;
  if (a.width == 4)
    pdl(k_packed_spmv_dot<4>, blocks(n), kBlock, 0, s, n, a.vals, a.offsets, a.diag, p, w, q, red,
        scalars, offset, status, epi);
  else
    pdl(k_packed_spmv_dot<8>, blocks(n), kBlock, 0, s, n, a.vals, a.offsets, a.diag, p, w, q, red,
        scalars, offset, status, epi);
}
void packed_smooth_dot2(int n, PackedRows a, const float* x, const float* b, const float* inv,
                        float* next, const float* q, DeviceReducer red, float* scalars,
                        int offset, int* status, Epilogue epi, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  if (a.width == 4)
    pdl(k_packed_smooth_dot2<4>, blocks(n), kBlock, 0, s, n, a.vals, a.offsets, a.diag, x, b, inv,
        next, q, red, scalars, offset, status, epi);
  else
    pdl(k_packed_smooth_dot2<8>, blocks(n), kBlock, 0, s, n, a.vals, a.offsets, a.diag, x, b, inv,
        next, q, red, scalars, offset, status, epi);
}
void coarse_solve(int count, const int* rows, const int* cols, const float* vals, float* x,
                  const float* b, const float* inv, const int* status, int sweeps,
                  cudaStream_t s) {
  ++counter;
  pdl(k_coarse_solve, 1, 32, 0, s, count, rows, cols, vals, x, b, inv, status, sweeps);
}
void diagonal(int n, const int* rows, const int* diag, const float* vals, float* inverse,
              int use_l1, DeviceReducer red, double* check, int slot, cudaStream_t s) {
  ++counter;
  pdl(k_diagonal, blocks(n), kBlock, 0, s, n, rows, diag, vals, inverse, use_l1, red, check, slot);
}
void prolong(int nf, const int* aggregate, const float* coarse, float* fine, const int* status,
             cudaStream_t s) {
  if (nf <= 0) return;
  ++counter;
  pdl(k_prolong, blocks(nf), kBlock, 0, s, nf, aggregate, coarse, fine, status);
}
void galerkin(int n_c, int nnz_c, const int* offsets, const int* entries, const unsigned* diagonal,
              const int* diag, bool diagonals, const float* fine, float* coarse, cudaStream_t s) {
  if (nnz_c <= 0) return;
  ++counter;
  const auto go = [&](auto kernel, int own) {
    pdl(kernel, own + blocks(nnz_c), kBlock, 0, s, n_c, nnz_c, offsets, entries, diagonal, diag,
        fine, coarse, own);
  };
  if (!diagonals)
    go(k_galerkin<Diagonals::Left>, 0);
  else if (nnz_c > kApartEntries)
    go(k_galerkin<Diagonals::Apart>, (n_c + kBlock - 1) / kBlock);
  else
    go(k_galerkin<Diagonals::Along>, 0);
}
void mark_diagonals(int n, const int* diag, unsigned* words, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_mark_diagonals, blocks(n), kBlock, 0, s, n, diag, words);
}
void m_matrix_diagonal(int nf, int nc, const int* offsets, const int* members, const int* fine_rows,
                       const int* fine_diag, const float* fine, const int* rows, const int* diag,
                       float* coarse, float* surplus, cudaStream_t s) {
  if (nc <= 0) return;
  ++counter;
  pdl(k_row_surplus, full_grid(nf), kBlock, 0, s, nf, fine_rows, fine_diag, fine, surplus);
  ++counter;
  pdl(k_m_matrix_combine, full_grid(nc), kBlock, 0, s, nc, offsets, members, surplus, rows, diag,
                                                      coarse);
}
void level_rows(int n, const int* rows, const int* diag, float* vals, const LevelRows& p,
                DeviceReducer red, double* check, int slot, cudaStream_t s) {
  ++counter;
  if (p.members != nullptr)
    pdl(k_level_rows<true>, blocks(n), kBlock, 0, s, n, rows, diag, vals, p.offsets, p.members,
        p.fine_surplus, p.inverse, p.surplus, p.store, red, check, slot);
  else
    pdl(k_level_rows<false>, blocks(n), kBlock, 0, s, n, rows, diag, vals, p.offsets, p.members,
        p.fine_surplus, p.inverse, p.surplus, p.store, red, check, slot);
}
void pcg_step_dot(int n, float* x, float* r, const float* p, const float* q, const int* rows,
                  const float* vals, const float* inv, float* next, DeviceReducer red,
                  float* scalars, int* status, cudaStream_t s) {
  ++counter;
  pdl(k_pcg_step_dot, blocks(n), kBlock, 0, s, n, x, r, p, q, rows, vals, inv, next, red, scalars,
      status);
}
void direction(int n, const float* z, float* p, const float* scalars, const int* status,
               cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_direction, blocks(n), kBlock, 0, s, n, z, p, scalars, status);
}
void bicg_direction(int n, const float* r, const float* v, float* p, const float* scalars,
                    const int* status, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_bicg_direction, blocks(n), kBlock, 0, s, n, r, v, p, scalars, status);
}
void bicg_difference(int n, const float* r, const float* q, float* sv, DeviceReducer red,
                     float* scalars, int* status, cudaStream_t s) {
  ++counter;
  pdl(k_bicg_difference, blocks(n), kBlock, 0, s, n, r, q, sv, red, scalars, status);
}
void bicg_step(int n, float* x, float* r, const float* z, const float* zs, const float* sv,
               const float* t, const float* shadow, DeviceReducer red, float* scalars, int* status,
               cudaStream_t s) {
  ++counter;
  pdl(k_bicg_step, blocks(n), kBlock, 0, s, n, x, r, z, zs, sv, t, shadow, red, scalars, status);
}
void multiply(int n, const float* r, const float* inverse, float* z, const int* status,
              cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_multiply, blocks(n), kBlock, 0, s, n, r, inverse, z, status);
}
void axpy(int n, float* y, const float* x, float a, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_axpy, blocks(n), kBlock, 0, s, n, y, x, a);
}
void fill(int n, float* x, float value, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_fill, blocks(n), kBlock, 0, s, n, x, value);
}
void reduce_into(ReduceMode mode, int n, const float* x, const float* y, const float* u,
                 const float* v, DeviceReducer red, float* scalars, int offset, int* status,
                 bool guard, Epilogue epi, cudaStream_t s) {
  ++counter;
  pdl(k_reduce_into, blocks(n), kBlock, 0, s, mode, n, x, y, u, v, red, scalars, offset, status,
                                             guard, epi);
}
void reduce_value(ReduceMode mode, int n, const float* x, const float* y, DeviceReducer red,
                  double* out, int slot, cudaStream_t s) {
  ++counter;
  pdl(k_reduce_value, blocks(n), kBlock, 0, s, mode, n, x, y, red, out, slot);
}
void solver_limits(float* scalars, float th, float tl, float dh, float dl, cudaStream_t s) {
  ++counter;
  pdl(k_solver_limits, 1, 32, 0, s, scalars, th, tl, dh, dl);
}
void solver_reset(float* scalars, int* status, int iterations, cudaStream_t s) {
  ++counter;
  pdl(k_solver_reset, 1, 1, 0, s, scalars, status, iterations);
}
void project(int n, float* x, const float* sum, float count_hi, float count_lo, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_project, blocks(n), kBlock, 0, s, n, x, sum, count_hi, count_lo);
}
void inner_alpha(float* scalars, int* status, const int* parent, int first, cudaStream_t s) {
  ++counter;
  pdl(k_inner_alpha, 1, 1, 0, s, scalars, status, parent, first);
}
void inner_first(int n, const float* b, const float* p, const float* q, float* x, float* t,
                 const float* scalars, const int* status, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_inner_first, blocks(n), kBlock, 0, s, n, b, p, q, x, t, scalars, status);
}
void inner_check(const float* scalars, int* status, cudaStream_t s) {
  ++counter;
  pdl(k_inner_check, 1, 1, 0, s, scalars, status);
}
void inner_beta(float* scalars, int* status, cudaStream_t s) {
  ++counter;
  pdl(k_inner_beta, 1, 1, 0, s, scalars, status);
}
void inner_step(int n, float* x, const float* p, const float* scalars, const int* status,
                cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_inner_step, blocks(n), kBlock, 0, s, n, x, p, scalars, status);
}

}  // namespace launch
}  // namespace kb2
