// Mixed-precision kernels (no reference counterpart): BF16 coarse operators,
// the dense FP64 coarsest-level inverse, and the FP64 refinement residual.
// Compiled with ordinary FMA contraction: these results are checked against the
// FP64 true residual, not by bitwise agreement with the reference.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "bf16_rows.cuh"
#include "common.cuh"
#include "inner_steps.cuh"
#include "kernels.hpp"

namespace kb2 {
namespace {
using namespace dev;

#define ROWS(i, n) \
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

inline int rows_grid(int n) {
  if (n >= (1 << 21)) return grid_for(n);
  return n > 0 ? (n + kBlock - 1) / kBlock : 1;
}

__device__ __forceinline__ float bf(unsigned short v) {
  return __bfloat162float(__ushort_as_bfloat16(v));
}

// Row scale = max |a_ij| (FP32); stored value = bf16(a_ij / scale).
__global__ void k_bf16_pack(int n, const float* __restrict__ vals, Bf16Store out) {
  pdl_entry();
  ROWS(i, n) bf16_store_row(i, vals, out);
}

// Whether a column lies further from its row than a 16-bit offset says.
__global__ void k_bf16_wide(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                            int* __restrict__ wide) {
  pdl_entry();
  bool found = false;
  ROWS(i, n) {
    for (int j = rows[i]; j < rows[i + 1]; ++j) found = found || abs(cols[j] - i) > 32767;
  }
  if (found) *wide = 1;
}

// Coarse rows hold about a dozen entries: four lanes share a row, each taking
// every fourth entry, so a warp reads eight rows' contiguous segments instead
// of 32 strided ones, and a row's dependent gathers are a quarter as long.
constexpr int kLanes = 4;
constexpr int kRowsPerWarp = 32 / kLanes;

// This lane's share of sum_j a_ij x_j (BF16 values, FP32 accumulation) of kR
// rows (-1: none). A row is taken in chunks of kLanes * kPerLane entries; a lane
// issues all its loads of a chunk, of kR rows, before any gather. These levels
// are bound by latency: a wave of warps waits for the row pointers, the entries
// and the gathered x in turn, so two rows per lane halve the number of waves
// where there are several (446,000 rows: a residual 11.7 us against 14.5, a
// sweep 11.1 against 13.7, the restriction to them 14.0 against 16.9); a level
// that fits in one wave is no faster for it, and the kernels with reductions,
// whose grid is fixed, slower (16.9 us against 15.9).
// kPacked: value and column offset in one word (launch::Bf16Rows), which is one
// load per entry instead of two and 4 bytes instead of 6.
constexpr int kPerLane = 3;
template <bool kPacked, int kR>
__device__ __forceinline__ void bf16_row_parts(const int (&row)[kR], int lane,
                                               const launch::Bf16Rows& m,
                                               const float* __restrict__ x, float (&acc)[kR]) {
  int at[kR], end[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    at[r] = row[r] >= 0 ? m.rows[row[r]] + lane : 0;
    end[r] = row[r] >= 0 ? m.rows[row[r] + 1] : 0;
    acc[r] = 0.0f;
  }
  while (at[0] < end[0] || at[kR - 1] < end[kR - 1]) {
    int c[kR][kPerLane];
    float a[kR][kPerLane], v[kR][kPerLane];
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
      for (int u = 0; u < kPerLane; ++u) {
        const int j = at[r] + u * kLanes;
        const bool in = j < end[r];
        if constexpr (kPacked) {
          const unsigned e = in ? __ldg(m.packed + j) : 0;
          c[r][u] = in ? row[r] + static_cast<short>(e & 0xffffu) : -1;
          a[r][u] = __uint_as_float(e & 0xffff0000u);
        } else {
          c[r][u] = in ? __ldg(m.cols + j) : -1;
          a[r][u] = in ? bf(__ldg(m.v16 + j)) : 0.0f;
        }
      }
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
      for (int u = 0; u < kPerLane; ++u) v[r][u] = c[r][u] >= 0 ? x[c[r][u]] : 0.0f;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
#pragma unroll
      for (int u = 0; u < kPerLane; ++u)
        if (c[r][u] >= 0) acc[r] = fmaf(a[r][u], v[r][u], acc[r]);
      at[r] += kLanes * kPerLane;
    }
  }
}
// Sum over the row's four lanes, in lane 0 (every lane of the warp calls it).
__device__ __forceinline__ float row_total(float v) {
  v += __shfl_down_sync(0xffffffffu, v, 2, kLanes);
  v += __shfl_down_sync(0xffffffffu, v, 1, kLanes);
  return v;
}

// Visits rows kLanes lanes at a time, kR rows (1 or 2) per group of lanes; the
// loop bound is uniform across a warp, so every lane reaches the shuffles.
// body(rows, lane), a row of -1 for none.
template <int kR, class Body>
__device__ __forceinline__ void for_rows(int n, Body body) {
  const int lane = threadIdx.x & (kLanes - 1);
  const int warp = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int warps = static_cast<int>((gridDim.x * blockDim.x) >> 5);
  for (int row0 = warp * kR * kRowsPerWarp; row0 < n; row0 += warps * kR * kRowsPerWarp) {
    int rows[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int i = row0 + r * kRowsPerWarp + static_cast<int>((threadIdx.x & 31) / kLanes);
      rows[r] = i < n ? i : -1;
    }
    body(rows, lane);
  }
}
// Rows above which the row kernels without a reduction take two per group: one
// wave of single rows (148 SMs x 2,048 threads / kLanes).
constexpr int kPairRows = 148 * 2048 / kLanes;

// A reduction's grid stays within the partials buffer (kMaxBlocks blocks).
inline int lanes_grid(int n, bool reduction) {
  const long long rows = reduction || n <= kPairRows ? n : (n + 1LL) / 2;
  const long long blocks = (rows * kLanes + kBlock - 1) / kBlock;
  const long long cap = reduction ? static_cast<long long>(kMaxBlocks) : (1LL << 30);
  return static_cast<int>(std::max(1LL, std::min(blocks, cap)));
}

// What a group's first lane needs besides the row's sum, loaded before it rather
// than a memory latency after it.
template <int kR>
struct RowData {
  float scale[kR], b[kR], inv[kR], x[kR];
  __device__ __forceinline__ RowData(const int (&rows)[kR], int lane, const launch::Bf16Rows& m,
                                     const float* __restrict__ right,
                                     const float* __restrict__ inverse,
                                     const float* __restrict__ iterate) {
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const bool mine = rows[r] >= 0 && lane == 0;
      scale[r] = mine ? m.scale[rows[r]] : 0.0f;
      b[r] = mine ? right[rows[r]] : 0.0f;
      inv[r] = mine && inverse ? inverse[rows[r]] : 0.0f;
      x[r] = mine && iterate ? iterate[rows[r]] : 0.0f;
    }
  }
  __device__ __forceinline__ float sweep(int r, float total) const {
    return x[r] + (2.0f / 3.0f) * inv[r] * (b[r] - scale[r] * total);
  }
};

// Damped L1-Jacobi sweep with the BF16 operator (FP32 accumulation).
template <bool kZero, bool kPacked, int kR>
__global__ void k_bf16_smooth(int n, launch::Bf16Rows m, const float* __restrict__ x,
                              const float* __restrict__ b, const float* __restrict__ inv,
                              float* __restrict__ next, const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  if (kZero) {
    ROWS(i, n) next[i] = (2.0f / 3.0f) * inv[i] * b[i];
    return;
  }
  for_rows<kR>(n, [&](const int (&rows)[kR], int lane) {
    const RowData<kR> d(rows, lane, m, b, inv, x);
    float acc[kR];
    bf16_row_parts<kPacked, kR>(rows, lane, m, x, acc);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const float total = row_total(acc[r]);
      if (rows[r] >= 0 && lane == 0) next[rows[r]] = d.sweep(r, total);
    }
  });
}

template <bool kPacked, int kR>
__global__ void k_bf16_residual(int n, launch::Bf16Rows m, const float* __restrict__ x,
                                const float* __restrict__ b, float* __restrict__ r,
                                const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  for_rows<kR>(n, [&](const int (&rows)[kR], int lane) {
    const RowData<kR> d(rows, lane, m, b, nullptr, nullptr);
    float acc[kR];
    bf16_row_parts<kPacked, kR>(rows, lane, m, x, acc);
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const float total = row_total(acc[q]);
      if (rows[q] >= 0 && lane == 0) r[rows[q]] = d.b[q] - d.scale[q] * total;
    }
  });
}

// Coarse b = sum of the fine residual over each aggregate's members, four
// lanes per aggregate with their member loads batched like the row kernels.
template <int kR>
__global__ void k_restrict_lanes(int nc, const int* __restrict__ offsets,
                                 const int* __restrict__ members, const float* __restrict__ fine,
                                 float* __restrict__ coarse, const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  for_rows<kR>(nc, [&](const int (&groups)[kR], int lane) {
    int at[kR], end[kR];
    float acc[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      at[r] = groups[r] >= 0 ? offsets[groups[r]] + lane : 0;
      end[r] = groups[r] >= 0 ? offsets[groups[r] + 1] : 0;
      acc[r] = 0.0f;
    }
    while (at[0] < end[0] || at[kR - 1] < end[kR - 1]) {
      int m[kR][kPerLane];
      float v[kR][kPerLane];
#pragma unroll
      for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int u = 0; u < kPerLane; ++u) {
          const int j = at[r] + u * kLanes;
          m[r][u] = j < end[r] ? members[j] : -1;
        }
#pragma unroll
      for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int u = 0; u < kPerLane; ++u) v[r][u] = m[r][u] >= 0 ? fine[m[r][u]] : 0.0f;
#pragma unroll
      for (int r = 0; r < kR; ++r) {
#pragma unroll
        for (int u = 0; u < kPerLane; ++u)
          if (m[r][u] >= 0) acc[r] += v[r][u];
        at[r] += kLanes * kPerLane;
      }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const float total = row_total(acc[r]);
      if (groups[r] >= 0 && lane == 0) coarse[groups[r]] = total;
    }
  });
}

// The last block stores the FP64 totals as (hi, lo) pairs at scalars[offset]
// and scalars[offset + 2]; returns true in its thread 0, which may then run the
// scalar step that follows (every block has read the status by then).
__device__ __forceinline__ bool finish_dot2(DeviceReducer red, double a, double b,
                                            float* scalars, int offset) {
  __shared__ double shared[32];
  a = block_sum(a, shared);
  b = block_sum(b, shared);
  const Reducer r{red.partials, red.ticket};
  if (!publish(r, a, b, true)) return false;
  const double total_a = gather(r, 0, shared);
  const double total_b = gather(r, 1, shared);
  if (threadIdx.x != 0) return false;
  store_pair(scalars, offset, total_a);
  store_pair(scalars, offset + 2, total_b);
  *r.ticket = 0;
  return true;
}

// K-cycle inner step on a BF16 level: q = A p and, in the same pass, the two
// products its step length needs, p.q and w.p -> scalars[0..3], then alpha.
// kFirst: p is the level's z, copied to `copy` on the way, `status` is the
// parent's, and the level's own status starts here (2, the plain cycle, while
// the parent has stopped); otherwise status is the level's own.
template <bool kFirst, bool kPacked>
__global__ void k_bf16_spmv_dot2(int n, launch::Bf16Rows m, const float* __restrict__ p,
                                 const float* __restrict__ w, float* __restrict__ q,
                                 float* __restrict__ copy, DeviceReducer red, float* scalars,
                                 const int* status, int* own) {
  pdl_entry();
  if (status[0] != 0) {
    if (kFirst && blockIdx.x == 0 && threadIdx.x == 0) own[0] = 2;
    return;
  }
  double a = 0.0, b = 0.0;
  for_rows<1>(n, [&](const int (&rows)[1], int lane) {
    const RowData<1> d(rows, lane, m, w, nullptr, p);
    float acc[1];
    bf16_row_parts<kPacked, 1>(rows, lane, m, p, acc);
#pragma unroll
    for (int r = 0; r < 1; ++r) {
      const float total = row_total(acc[r]);
      if (rows[r] < 0 || lane != 0) continue;
      const float qi = d.scale[r] * total, pi = d.x[r];
      q[rows[r]] = qi;
      if (kFirst) copy[rows[r]] = pi;
      a += static_cast<double>(pi) * static_cast<double>(qi);
      b += static_cast<double>(d.b[r]) * static_cast<double>(pi);
    }
  });
  if (!finish_dot2(red, a, b, scalars, 0)) return;
  if (kFirst) own[0] = 0;
  inner_alpha(scalars, own, kFirst);
}

// The last sweep of the second inner cycle with z.q -> scalars[4..5] (q = A p of
// the first) and beta.
template <bool kPacked>
__global__ void k_bf16_smooth_dot(int n, launch::Bf16Rows m, const float* __restrict__ x,
                                  const float* __restrict__ b, const float* __restrict__ inv,
                                  float* __restrict__ next, const float* __restrict__ q,
                                  DeviceReducer red, float* scalars, int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  double a = 0.0;
  for_rows<1>(n, [&](const int (&rows)[1], int lane) {
    const RowData<1> d(rows, lane, m, b, inv, x);
    float acc[1];
    bf16_row_parts<kPacked, 1>(rows, lane, m, x, acc);
#pragma unroll
    for (int r = 0; r < 1; ++r) {
      const float total = row_total(acc[r]);
      if (rows[r] < 0 || lane != 0) continue;
      const float z = d.sweep(r, total);
      next[rows[r]] = z;
      a += static_cast<double>(z) * static_cast<double>(q[rows[r]]);
    }
  });
  __shared__ double shared[32];
  a = block_sum(a, shared);
  const Reducer r{red.partials, red.ticket};
  if (!publish(r, a, 0.0, false)) return;
  const double total = gather(r, 0, shared);
  if (threadIdx.x != 0) return;
  store_pair(scalars, 4, total);
  *r.ticket = 0;
  inner_beta(scalars, status);
}

// amg_inner_first with the next reduction fused: x = alpha p, t = b - alpha q
// (or x = p, t = 0 when the level's status is not running), then t.t and b.b
// -> scalars[4..7] and the exit check. Skipped (reduction included) while
// status[0] != 0, as every reader of those slots is.
__global__ void k_inner_first_dot(int n, const float* __restrict__ b, const float* __restrict__ p,
                                  const float* __restrict__ q, float* __restrict__ x,
                                  float* __restrict__ t, float* scalars, int* status,
                                  DeviceReducer red) {
  pdl_entry();
  const bool running = status[0] == 0;
  const float alpha = kp_float(kp_load(scalars, 8));
  double tt = 0.0, bb = 0.0;
  ROWS(i, n) {
    const float ti = running ? b[i] - alpha * q[i] : 0.0f;
    x[i] = running ? alpha * p[i] : p[i];
    t[i] = ti;
    tt += static_cast<double>(ti) * static_cast<double>(ti);
    bb += static_cast<double>(b[i]) * static_cast<double>(b[i]);
  }
  if (!running) return;
  if (finish_dot2(red, tt, bb, scalars, 4)) inner_check(scalars, status);
}

// Dense FP64 Cholesky of the coarsest operator and its explicit inverse for
// kPackedDense < n <= 1024, blocked in 32 x 32 blocks and spread over many
// CTAs (a sequence of launches at refresh time). L is n x n row-major scratch
// in global memory (2 MB at n = 512, L2-resident) and W the n x n inverse.
//   1. L = the lower triangle of A (the strict upper triangle is free; the
//      original diagonal is kept there for the pivot ratio: a_kk at L[k][n-1],
//      a_{n-1,n-1} at L[0][n-2]);
//   2. per 32-column panel: the diagonal block factored in one CTA (shared
//      memory), the rows below solved against it (a thread per row), the
//      trailing lower triangle updated tile by tile (a CTA per 32 x 32 tile);
//   3. X = L^-1 into W's lower triangle: the diagonal blocks inverted in
//      parallel, then block diagonal d = 1, 2, ...: X_ij = -X_ii sum_{k=j}^{i-1}
//      L_ik X_kj for i - j = d, a CTA per block;
//   4. W = X^T X tile by tile into L's buffer, then copied to W.
// Every element is summed in a fixed order, so the result is deterministic.
// *error = 1 if a pivot was not positive (it is replaced by 1 so the kernels
// finish), else 0; with `ratio`, *ratio is the smallest pivot relative to its
// row's original diagonal (0 if one failed).
constexpr int kNb = 32;                         // block size
constexpr int kNbThreads = kNb * kNb;           // one thread per block element

__device__ __forceinline__ std::size_t at(int n, int i, int j) {
  return static_cast<std::size_t>(i) * n + j;
}
// Where row k's original diagonal is kept (strict upper triangle of L).
__device__ __forceinline__ std::size_t diag_slot(int n, int k) {
  return k < n - 1 ? at(n, k, n - 1) : at(n, 0, n - 2);
}

__global__ void k_dense_zero(std::size_t count, double* __restrict__ L) {
  pdl_entry();
  for (std::size_t k = blockIdx.x * static_cast<std::size_t>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<std::size_t>(gridDim.x) * blockDim.x)
    L[k] = 0.0;
}

__global__ void k_dense_scatter(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                                const float* __restrict__ vals, double* __restrict__ L,
                                double* error, double* ratio) {
  pdl_entry();
  ROWS(i, n) {
    for (int j = rows[i]; j < rows[i + 1]; ++j) {
      const int c = cols[j];
      if (c <= i) L[at(n, i, c)] = vals[j];
      if (c == i) L[diag_slot(n, i)] = vals[j];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *error = 0.0;
    if (ratio) *ratio = 1.0;
  }
}

// Factor the diagonal block of panel k0 (b = min(32, n - k0) columns) in place.
__global__ void __launch_bounds__(kNbThreads)
    k_dense_panel_factor(int n, int k0, double* __restrict__ L, double* error, double* ratio) {
  pdl_entry();
  __shared__ double D[kNb][kNb + 1];
  const int b = min(kNb, n - k0);
  const int r = threadIdx.x / kNb, c = threadIdx.x % kNb;
  if (r < b && c <= r) D[r][c] = L[at(n, k0 + r, k0 + c)];
  __syncthreads();
  for (int k = 0; k < b; ++k) {
    if (threadIdx.x == 0) {
      double d = D[k][k];
      if (!(d > 0.0)) {
        *error = 1.0;
        if (ratio) *ratio = 0.0;
        d = 1.0;
      } else if (ratio && *error == 0.0) {
        *ratio = fmin(*ratio, d / L[diag_slot(n, k0 + k)]);
      }
      D[k][k] = sqrt(d);
    }
    __syncthreads();
    if (c == k && r > k && r < b) D[r][k] /= D[k][k];
    __syncthreads();
    if (r < b && c > k && c <= r) D[r][c] -= D[r][k] * D[c][k];
    __syncthreads();
  }
  if (r < b && c <= r) L[at(n, k0 + r, k0 + c)] = D[r][c];
}

// The rows below panel k0: x L_kk^T = a for each row's panel slice x.
__global__ void k_dense_panel_solve(int n, int k0, double* __restrict__ L) {
  pdl_entry();
  __shared__ double D[kNb][kNb + 1];
  const int b = min(kNb, n - k0);
  for (int e = threadIdx.x; e < kNb * kNb; e += blockDim.x) {
    const int r = e / kNb, c = e % kNb;
    D[r][c] = r < b && c <= r ? L[at(n, k0 + r, k0 + c)] : 0.0;
  }
  __syncthreads();
  const int i = k0 + b + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double x[kNb];
#pragma unroll
  for (int c = 0; c < kNb; ++c) x[c] = c < b ? L[at(n, i, k0 + c)] : 0.0;
#pragma unroll
  for (int c = 0; c < kNb; ++c) {
    if (c >= b) break;
    double v = x[c];
    for (int m = 0; m < c; ++m) v -= x[m] * D[c][m];
    x[c] = v / D[c][c];
  }
#pragma unroll
  for (int c = 0; c < kNb; ++c)
    if (c < b) L[at(n, i, k0 + c)] = x[c];
}

// Trailing update below panel k0: L_ij -= sum_c L_ic L_jc over the panel's
// columns, for j <= i in the rows after the panel. Block (bx, by) of the
// grid is tile (ti, tj) = (by, bx) of the trailing part; tiles above the
// diagonal do nothing.
__global__ void __launch_bounds__(kNbThreads)
    k_dense_panel_update(int n, int k0, double* __restrict__ L) {
  pdl_entry();
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  __shared__ double Pi[kNb][kNb + 1], Pj[kNb][kNb + 1];
  const int b = min(kNb, n - k0);
  const int base = k0 + b;
  const int r = threadIdx.x / kNb, c = threadIdx.x % kNb;
  const int i0 = base + ti * kNb, j0 = base + tj * kNb;
  Pi[r][c] = i0 + r < n && c < b ? L[at(n, i0 + r, k0 + c)] : 0.0;
  Pj[r][c] = j0 + r < n && c < b ? L[at(n, j0 + r, k0 + c)] : 0.0;
  __syncthreads();
  const int i = i0 + r, j = j0 + c;
  if (i >= n || j >= n || j > i) return;
  double sum = 0.0;
  for (int m = 0; m < b; ++m) sum += Pi[r][m] * Pj[c][m];
  L[at(n, i, j)] -= sum;
}

// X_pp = L_pp^-1 for every diagonal block p (a CTA each), into W.
__global__ void __launch_bounds__(kNbThreads)
    k_dense_block_inverse(int n, const double* __restrict__ L, double* __restrict__ W) {
  pdl_entry();
  __shared__ double D[kNb][kNb + 1], X[kNb][kNb + 1];
  const int k0 = blockIdx.x * kNb;
  const int b = min(kNb, n - k0);
  const int r = threadIdx.x / kNb, c = threadIdx.x % kNb;
  D[r][c] = r < b && c <= r ? L[at(n, k0 + r, k0 + c)] : 0.0;
  X[r][c] = 0.0;
  __syncthreads();
  // Column c of X: L_pp X[:, c] = e_c, forward substitution by thread (0, c).
  if (r == 0 && c < b) {
    for (int i = c; i < b; ++i) {
      double v = i == c ? 1.0 : 0.0;
      for (int m = c; m < i; ++m) v -= D[i][m] * X[m][c];
      X[i][c] = v / D[i][i];
    }
  }
  __syncthreads();
  if (r < b && c <= r) W[at(n, k0 + r, k0 + c)] = X[r][c];
}

// Block diagonal d of X: X_ij = -X_ii sum_{k=j}^{i-1} L_ik X_kj, i = j + d
// (block indices), a CTA per j.
__global__ void __launch_bounds__(kNbThreads)
    k_dense_block_offdiag(int n, int d, const double* __restrict__ L, double* __restrict__ W) {
  pdl_entry();
  __shared__ double A[kNb][kNb + 1], B[kNb][kNb + 1];
  const int jb = blockIdx.x, ib = jb + d;
  const int i0 = ib * kNb, j0 = jb * kNb;
  const int r = threadIdx.x / kNb, c = threadIdx.x % kNb;
  double sum = 0.0;  // S[r][c]
  for (int kb = jb; kb < ib; ++kb) {
    const int k0 = kb * kNb;
    // A = L_ik (rows i0.., columns k0..), B = X_kj (rows k0.., columns j0..);
    // X_kj is lower triangular when k == j.
    A[r][c] = i0 + r < n ? L[at(n, i0 + r, k0 + c)] : 0.0;
    B[r][c] = k0 + r < n && (kb > jb || c <= r) ? W[at(n, k0 + r, j0 + c)] : 0.0;
    __syncthreads();
    for (int m = 0; m < kNb; ++m) sum += A[r][m] * B[m][c];
    __syncthreads();
  }
  // X_ij = -X_ii S, X_ii lower triangular.
  A[r][c] = i0 + r < n && c <= r ? W[at(n, i0 + r, i0 + c)] : 0.0;
  B[r][c] = sum;
  __syncthreads();
  double x = 0.0;
  for (int m = 0; m <= r; ++m) x -= A[r][m] * B[m][c];
  if (i0 + r < n && j0 + c < n) W[at(n, i0 + r, j0 + c)] = x;
}

// Tile (ti, tj), tj <= ti, of W = X^T X: sum over block rows k >= ti of
// X_k,ti^T X_k,tj (X lower triangular in W), into out (both (i, j) and (j, i)).
__global__ void __launch_bounds__(kNbThreads)
    k_dense_gram(int n, const double* __restrict__ X, double* __restrict__ out) {
  pdl_entry();
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  __shared__ double A[kNb][kNb + 1], B[kNb][kNb + 1];
  const int nb = (n + kNb - 1) / kNb;
  const int r = threadIdx.x / kNb, c = threadIdx.x % kNb;
  const int i = ti * kNb + r, j = tj * kNb + c;
  double sum = 0.0;
  for (int kb = ti; kb < nb; ++kb) {
    const int k0 = kb * kNb;
    // A[m][r] = X[k0 + m][ti*32 + r], B[m][c] = X[k0 + m][tj*32 + c] (zero above the diagonal).
    const int kr = k0 + r;
    A[r][c] = kr < n && ti * kNb + c < n && ti * kNb + c <= kr ? X[at(n, kr, ti * kNb + c)] : 0.0;
    B[r][c] = kr < n && tj * kNb + c < n && tj * kNb + c <= kr ? X[at(n, kr, tj * kNb + c)] : 0.0;
    __syncthreads();
    for (int m = 0; m < kNb; ++m) sum += A[m][r] * B[m][c];
    __syncthreads();
  }
  if (i < n && j < n) {
    out[at(n, i, j)] = sum;
    out[at(n, j, i)] = sum;
  }
}

__global__ void k_dense_copy(std::size_t count, const double* __restrict__ from,
                             double* __restrict__ to) {
  pdl_entry();
  for (std::size_t k = blockIdx.x * static_cast<std::size_t>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<std::size_t>(gridDim.x) * blockDim.x)
    to[k] = from[k];
}

// The inverse for n <= kSharedDense in one CTA: the root-free factorisation
// A = L D L^T and X = L^-1 in one elimination, then W = X^T D^-1 X (symmetric).
// Its length is the n dependent steps, so each step is kept short: warp w's lane
// l holds elements (w + 32 a, l + 32 c) in registers (A right of the diagonal
// step, X left of it), and a step needs one division, the current column of A and
// the current row of X, which their owners put into shared memory as they
// update them for the next step, and one barrier. `L` (global) is not used. (A
// Cholesky factor and a separate substitution in shared memory, five barriers,
// a root and a column of divisions per step, took 231 us at 107 rows; this 118.)
constexpr int kSharedDense = 112;
constexpr int kDenseThreads = 1024;
constexpr int kDenseTile = 4;  // elements of a thread in each direction
static_assert(32 * kDenseTile >= kSharedDense, "a thread's rows and columns");

// Lower-triangle pair number p -> (i, j), j <= i, rows counted from 0.
__device__ __forceinline__ void triangle_pair(int p, int& i, int& j) {
  i = static_cast<int>((sqrt(8.0 * p + 1.0) - 1.0) * 0.5);
  while ((i + 1) * (i + 2) / 2 <= p) ++i;
  while (i * (i + 1) / 2 > p) --i;
  j = p - i * (i + 1) / 2;
}

// The lower triangle of the operator into `dense` (n x n) and its diagonal into
// diag0; all threads of the block, which the caller synchronises before and after.
__device__ __forceinline__ void dense_lower(int n, const int* __restrict__ rows,
                                            const int* __restrict__ cols,
                                            const float* __restrict__ vals, double* dense,
                                            double* diag0) {
  for (int k = threadIdx.x; k < n * n; k += kDenseThreads) dense[k] = 0.0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kDenseThreads)
    for (int j = rows[i]; j < rows[i + 1]; ++j) {
      if (cols[j] <= i) dense[i * n + cols[j]] = vals[j];
      if (cols[j] == i) diag0[i] = vals[j];
    }
}

// The pivots of the Cholesky factor of `dense`, each element updated in the order
// of the steps k: thread 0's `failed` (a pivot is not positive) and `smallest` (the
// least share of its diagonal). Below this share the root-free elimination's
// rounding may give a vanishing pivot another sign than the factor's, on which the
// caller's refusal of an operator that is not SPD rests: a 4 x 5 Neumann Laplacian
// has a positive last pivot in the factor and a negative one in the elimination.
// The inverse of such an operator is not used for solves (Solver::choose_coarsest
// asks for the same share).
constexpr double kConditionedPivot = 1e-6;
__device__ void cholesky_pivots(int n, double* dense, const double* diag0, double* column,
                                bool& failed, double& smallest) {
  __shared__ double pivot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  failed = false;
  smallest = 1.0;
  for (int k = 0; k < n; ++k) {
    if (threadIdx.x == 0) {
      double d = dense[k * n + k];
      if (!(d > 0.0)) {
        failed = true;
        d = 1.0;
      } else {
        smallest = fmin(smallest, d / diag0[k]);
      }
      pivot = sqrt(d);
    }
    __syncthreads();
    for (int i = k + 1 + static_cast<int>(threadIdx.x); i < n; i += kDenseThreads)
      column[i] = dense[i * n + k] / pivot;
    __syncthreads();
    for (int i = k + 1 + warp; i < n; i += kDenseThreads / 32)
      for (int j = k + 1 + lane; j <= i; j += 32)
        dense[i * n + j] = fma(-column[i], column[j], dense[i * n + j]);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kDenseThreads)
    k_dense_inverse_shared(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                           const float* __restrict__ vals, double* __restrict__ W, double* error,
                           double* ratio) {
  pdl_entry();
  extern __shared__ double dense[];  // n x n
  __shared__ double column[2][kSharedDense], row[2][kSharedDense];
  __shared__ double inverse[kSharedDense], diag0[kSharedDense];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  bool failed = false;
  double smallest = 1.0;  // thread 0's
  dense_lower(n, rows, cols, vals, dense, diag0);
  __syncthreads();
  double m[kDenseTile][kDenseTile];
#pragma unroll
  for (int a = 0; a < kDenseTile; ++a)
#pragma unroll
    for (int c = 0; c < kDenseTile; ++c) {
      const int i = warp + 32 * a, j = lane + 32 * c;
      m[a][c] = i < n && j <= i ? dense[i * n + j] : 0.0;
      if (c == 0 && lane == 0 && i < n) column[0][i] = m[a][0];
    }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const int now = k & 1, next = now ^ 1;
    double d = column[now][k];
    const bool positive = d > 0.0;
    if (t == 0) {
      if (positive) smallest = fmin(smallest, d / diag0[k]);
      else failed = true;
    }
    if (!positive) d = 1.0;
    const double inv = 1.0 / d;
    if (t == 0) inverse[k] = inv;
    double s[kDenseTile];
#pragma unroll
    for (int c = 0; c < kDenseTile; ++c) {
      const int j = lane + 32 * c;
      s[c] = j >= n || j == k ? 0.0 : j < k ? row[now][j] : column[now][j];
    }
#pragma unroll
    for (int a = 0; a < kDenseTile; ++a) {
      const int i = warp + 32 * a;
      if (i <= k || i >= n) continue;
      const double f = column[now][i] * inv;
#pragma unroll
      for (int c = 0; c < kDenseTile; ++c) {
        const int j = lane + 32 * c;
        if (j > i) continue;
        m[a][c] = j == k ? -f : fma(-f, s[c], m[a][c]);
        if (j == k + 1) column[next][i] = m[a][c];
        if (i == k + 1 && j <= k) row[next][j] = m[a][c];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < kDenseTile; ++a)
#pragma unroll
    for (int c = 0; c < kDenseTile; ++c) {
      const int i = warp + 32 * a, j = lane + 32 * c;
      if (i < n && j < n) dense[i * n + j] = j < i ? m[a][c] : j == i ? 1.0 : 0.0;
    }
  __syncthreads();
  // W_ij = sum_{k >= i} X_ki X_kj / d_k for j <= i, a warp per row i.
  for (int i = warp; i < n; i += 32) {
    double acc[kDenseTile] = {};
    for (int k = i; k < n; ++k) {
      const double f = dense[k * n + i] * inverse[k];
#pragma unroll
      for (int c = 0; c < kDenseTile; ++c)
        if (lane + 32 * c <= i) acc[c] = fma(f, dense[k * n + lane + 32 * c], acc[c]);
    }
#pragma unroll
    for (int c = 0; c < kDenseTile; ++c) {
      const int j = lane + 32 * c;
      if (j > i) continue;
      W[static_cast<std::size_t>(i) * n + j] = acc[c];
      W[static_cast<std::size_t>(j) * n + i] = acc[c];
    }
  }
  if (__syncthreads_or(t == 0 && (failed || smallest < kConditionedPivot))) {
    dense_lower(n, rows, cols, vals, dense, diag0);
    __syncthreads();
    cholesky_pivots(n, dense, diag0, inverse, failed, smallest);
  }
  if (t == 0) {
    *error = failed ? 1.0 : 0.0;
    if (ratio) *ratio = failed ? 0.0 : smallest;
  }
}

// The same for kSharedDense < n <= kPackedDense: only the lower triangle, packed
// (row i at i (i + 1) / 2), fits in shared memory, so L is inverted in place.
// Column j of X = L^-1 (j from the right) needs the already inverted columns
// k > j and column j of L: X_ij = -(sum_{k=j+1..i} X_ik L_kj) / L_jj, one warp
// per row i with the sum split over the lanes; then W = X^T X.
constexpr int kPackedDense = 236;  // (n (n + 1) / 2 + 2 n) doubles <= 227 KB
constexpr int kPackedThreads = 1024;

__device__ __forceinline__ int packed(int i, int j) { return i * (i + 1) / 2 + j; }

__global__ void __launch_bounds__(kPackedThreads)
    k_dense_inverse_packed(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                           const float* __restrict__ vals, double* __restrict__ W, double* error,
                           double* ratio) {
  pdl_entry();
  extern __shared__ double dense[];
  const int total = n * (n + 1) / 2;
  double* P = dense;           // packed lower triangle: L, then X = L^-1
  double* temp = P + total;    // one column's new entries
  double* diag0 = temp + n;    // the input diagonal
  const int t = threadIdx.x, T = blockDim.x, lane = t & 31, warp = t >> 5, warps = T >> 5;
  __shared__ int failed;
  __shared__ double smallest, pivot;
  if (t == 0) {
    failed = 0;
    smallest = 1.0;
  }
  for (int k = t; k < total; k += T) P[k] = 0.0;
  __syncthreads();
  for (int i = t; i < n; i += T)
    for (int j = rows[i]; j < rows[i + 1]; ++j) {
      if (cols[j] <= i) P[packed(i, cols[j])] = vals[j];
      if (cols[j] == i) diag0[i] = vals[j];
    }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    if (t == 0) {
      double d = P[packed(k, k)];
      if (!(d > 0.0)) {
        failed = 1;
        d = 1.0;
      } else {
        smallest = fmin(smallest, d / diag0[k]);
      }
      pivot = sqrt(d);
      P[packed(k, k)] = pivot;
    }
    __syncthreads();
    for (int i = k + 1 + t; i < n; i += T) P[packed(i, k)] /= pivot;
    __syncthreads();
    const int m = n - k - 1;
    for (int p = t; p < m * (m + 1) / 2; p += T) {
      int a, b;
      triangle_pair(p, a, b);
      const int i = k + 1 + a, j = k + 1 + b;
      P[packed(i, j)] -= P[packed(i, k)] * P[packed(j, k)];
    }
    __syncthreads();
  }
  for (int j = n - 1; j >= 0; --j) {
    const double ljj = P[packed(j, j)];  // read before this step's writes
    for (int i = j + 1 + warp; i < n; i += warps) {
      double acc = 0.0;
      for (int k = j + 1 + lane; k <= i; k += 32) acc += P[packed(i, k)] * P[packed(k, j)];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d);
      if (lane == 0) temp[i] = acc;
    }
    __syncthreads();
    for (int i = j + 1 + t; i < n; i += T) P[packed(i, j)] = -temp[i] / ljj;
    if (t == 0) P[packed(j, j)] = 1.0 / ljj;
    __syncthreads();
  }
  for (int p = t; p < total; p += T) {
    int i, j;
    triangle_pair(p, i, j);
    double acc = 0.0;
    for (int k = i; k < n; ++k) acc += P[packed(k, i)] * P[packed(k, j)];
    W[static_cast<std::size_t>(i) * n + j] = acc;
    W[static_cast<std::size_t>(j) * n + i] = acc;
  }
  if (t == 0) {
    *error = failed ? 1.0 : 0.0;
    if (ratio) *ratio = failed ? 0.0 : smallest;
  }
}

// x = A^-1 b with the dense FP64 inverse: one warp per row, FP64 accumulation.
__global__ void k_dense_solve(int n, const double* __restrict__ W, const float* __restrict__ b,
                              float* __restrict__ x, const int* __restrict__ status) {
  pdl_entry();
  if (status[0] != 0) return;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int i = warp; i < n; i += warps) {
    double acc = 0.0;
    const double* row = W + static_cast<std::size_t>(i) * n;
    for (int k = lane; k < n; k += 32) acc += row[k] * static_cast<double>(b[k]);
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d);
    if (lane == 0) x[i] = static_cast<float>(acc);
  }
}

// FP64 refinement residual: r = b - A x in FP64 (x FP64, A and b FP32), written
// rounded to FP32 for the inner solve, with ||r||^2 reduced in FP64 into out[slot].
__global__ void k_residual64(int n, const int* __restrict__ rows, const int* __restrict__ cols,
                             const float* __restrict__ vals, const double* __restrict__ x,
                             const float* __restrict__ b, float* __restrict__ rf,
                             DeviceReducer red, double* out, int slot) {
  pdl_entry();
  double acc = 0.0;
  ROWS(i, n) {
    double s = static_cast<double>(b[i]);
    const int end = rows[i + 1];
    for (int j = rows[i]; j < end; ++j) s -= static_cast<double>(vals[j]) * x[cols[j]];
    rf[i] = static_cast<float>(s);
    acc += s * s;
  }
  __shared__ double shared[32];
  acc = block_sum(acc, shared);
  const Reducer r{red.partials, red.ticket};
  if (!publish(r, acc, 0, false)) return;
  const double total = gather(r, 0, shared);
  if (threadIdx.x == 0) {
    out[slot] = total;
    *r.ticket = 0;
  }
}

__global__ void k_update64(int n, double* __restrict__ x, const float* __restrict__ e) {
  pdl_entry();
  ROWS(i, n) x[i] += static_cast<double>(e[i]);
}

__global__ void k_widen(int n, const float* __restrict__ x, double* __restrict__ y) {
  pdl_entry();
  ROWS(i, n) y[i] = static_cast<double>(x[i]);
}

__global__ void k_narrow(int n, const double* __restrict__ y, float* __restrict__ x) {
  pdl_entry();
  ROWS(i, n) x[i] = static_cast<float>(y[i]);
}

}  // namespace

namespace launch {

void bf16_pack(int n, const float* vals, const Bf16Store& out, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_bf16_pack, rows_grid(n), kBlock, 0, s, n, vals, out);
}
void bf16_wide(int n, const int* rows, const int* cols, int* wide, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_bf16_wide, rows_grid(n), kBlock, 0, s, n, rows, cols, wide);
}
void bf16_smooth(int n, const Bf16Rows& m, const float* x, const float* b, const float* inv,
                 float* next, const int* status, bool zero_start, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  if (zero_start)
    pdl(k_bf16_smooth<true, false, 1>, rows_grid(n), kBlock, 0, s, n, m, x, b, inv, next, status);
  else
    pdl(m.packed != nullptr
            ? (n > kPairRows ? k_bf16_smooth<false, true, 2> : k_bf16_smooth<false, true, 1>)
            : (n > kPairRows ? k_bf16_smooth<false, false, 2> : k_bf16_smooth<false, false, 1>),
        lanes_grid(n, false), kBlock, 0, s, n, m, x, b, inv, next, status);
}
void restrict_lanes(int nc, const int* offsets, const int* members, const float* fine,
                    float* coarse, const int* status, cudaStream_t s) {
  if (nc <= 0) return;
  ++counter;
  pdl(nc > kPairRows ? k_restrict_lanes<2> : k_restrict_lanes<1>, lanes_grid(nc, false), kBlock, 0,
      s, nc, offsets, members, fine, coarse, status);
}
void bf16_spmv_dot2(int n, const Bf16Rows& m, const float* p, const float* w, float* q, float* copy,
                    DeviceReducer red, float* scalars, const int* parent, int* status,
                    cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  const auto go = [&](auto kernel, const int* guard) {
    pdl(kernel, lanes_grid(n, true), kBlock, 0, s, n, m, p, w, q, copy, red, scalars, guard, status);
  };
  const bool packed = m.packed != nullptr;
  if (copy != nullptr)
    go(packed ? k_bf16_spmv_dot2<true, true> : k_bf16_spmv_dot2<true, false>, parent);
  else
    go(packed ? k_bf16_spmv_dot2<false, true> : k_bf16_spmv_dot2<false, false>, status);
}
void bf16_smooth_dot(int n, const Bf16Rows& m, const float* x, const float* b, const float* inv,
                     float* next, const float* q, DeviceReducer red, float* scalars, int* status,
                     cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(m.packed != nullptr ? k_bf16_smooth_dot<true> : k_bf16_smooth_dot<false>, lanes_grid(n, true),
      kBlock, 0, s, n, m, x, b, inv, next, q, red, scalars, status);
}
void inner_first_dot(int n, const float* b, const float* p, const float* q, float* x, float* t,
                     float* scalars, int* status, DeviceReducer red, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_inner_first_dot, grid_for(n), kBlock, 0, s, n, b, p, q, x, t, scalars, status, red);
}
void bf16_residual(int n, const Bf16Rows& m, const float* x, const float* b, float* r,
                   const int* status, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(m.packed != nullptr ? (n > kPairRows ? k_bf16_residual<true, 2> : k_bf16_residual<true, 1>)
                          : (n > kPairRows ? k_bf16_residual<false, 2> : k_bf16_residual<false, 1>),
      lanes_grid(n, false), kBlock, 0, s, n, m, x, b, r, status);
}
void dense_inverse(int n, const int* rows, const int* cols, const float* vals, double* lower,
                   double* inverse, double* error, cudaStream_t s, double* ratio) {
  if (n <= 0) return;
  ++counter;
  if (n <= kSharedDense) {
    const int bytes = n * n * static_cast<int>(sizeof(double));
    static std::atomic<unsigned long long> raised{0};
    raise_shared_limit(reinterpret_cast<const void*>(k_dense_inverse_shared),
                       kSharedDense * kSharedDense * static_cast<int>(sizeof(double)), raised);
    pdl(k_dense_inverse_shared, 1, kDenseThreads, bytes, s, n, rows, cols, vals, inverse, error,
                                                            ratio);
    return;
  }
  if (n <= kPackedDense) {
    const int bytes = (n * (n + 1) / 2 + 2 * n) * static_cast<int>(sizeof(double));
    static std::atomic<unsigned long long> raised_packed{0};
    raise_shared_limit(
        reinterpret_cast<const void*>(k_dense_inverse_packed),
        (kPackedDense * (kPackedDense + 1) / 2 + 2 * kPackedDense) * static_cast<int>(sizeof(double)),
        raised_packed);
    pdl(k_dense_inverse_packed, 1, kPackedThreads, bytes, s, n, rows, cols, vals, inverse, error,
                                                            ratio);
    return;
  }
  // Blocked, over many CTAs (see k_dense_panel_factor and the kernels after it).
  const std::size_t count = static_cast<std::size_t>(n) * n;
  const int nb = (n + kNb - 1) / kNb;
  const int fill = static_cast<int>(std::min<std::size_t>((count + kBlock - 1) / kBlock, 1184));
  counter += 4 * nb + 2;
  pdl(k_dense_zero, fill, kBlock, 0, s, count, lower);
  pdl(k_dense_scatter, (n + kBlock - 1) / kBlock, kBlock, 0, s, n, rows, cols, vals, lower, error,
      ratio);
  for (int p = 0; p < nb; ++p) {
    const int k0 = p * kNb;
    pdl(k_dense_panel_factor, 1, kNbThreads, 0, s, n, k0, lower, error, ratio);
    const int below = n - k0 - kNb;
    if (below > 0) {
      pdl(k_dense_panel_solve, (below + 127) / 128, 128, 0, s, n, k0, lower);
      const int tiles = (below + kNb - 1) / kNb;
      pdl(k_dense_panel_update, dim3(tiles, tiles), kNbThreads, 0, s, n, k0, lower);
    }
  }
  pdl(k_dense_block_inverse, nb, kNbThreads, 0, s, n, static_cast<const double*>(lower), inverse);
  for (int d = 1; d < nb; ++d)
    pdl(k_dense_block_offdiag, nb - d, kNbThreads, 0, s, n, d, static_cast<const double*>(lower),
        inverse);
  pdl(k_dense_gram, dim3(nb, nb), kNbThreads, 0, s, n, static_cast<const double*>(inverse), lower);
  pdl(k_dense_copy, fill, kBlock, 0, s, count, static_cast<const double*>(lower), inverse);
}
void dense_solve(int n, const double* inverse, const float* b, float* x, const int* status,
                 cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  const int blocks = std::min(1184, (n * 32 + kBlock - 1) / kBlock);
  pdl(k_dense_solve, blocks, kBlock, 0, s, n, inverse, b, x, status);
}
void residual64(int n, const int* rows, const int* cols, const float* vals, const double* x,
                const float* b, float* rf, DeviceReducer red, double* out, int slot,
                cudaStream_t s) {
  ++counter;
  pdl(k_residual64, grid_for(n), kBlock, 0, s, n, rows, cols, vals, x, b, rf, red, out, slot);
}
void update64(int n, double* x, const float* e, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_update64, rows_grid(n), kBlock, 0, s, n, x, e);
}
void widen(int n, const float* x, double* y, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_widen, rows_grid(n), kBlock, 0, s, n, x, y);
}
void narrow(int n, const double* y, float* x, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_narrow, rows_grid(n), kBlock, 0, s, n, y, x);
}

}  // namespace launch
}  // namespace kb2
