// Row kernels of the plain (reference-parity) coarse levels for sm_100a
// (compiled with --fmad=false): the damped L1-Jacobi sweep, the compensated
// residual, the transfers and the small levels' whole V-cycle, with the same
// float operations in the same order per row as exact_kernels.cu.
//
// A coarse level is latency-bound: a few thousand to a few hundred thousand
// rows whose operator sits in L2, with rows of 5 to 200 entries. A thread per
// row walks its entries one by one (column, then the gathered x, then some
// twenty dependent float operations), and a warp waits for its longest row.
// Here a block takes kRows consecutive rows, whose entries are consecutive in
// the CSR arrays: all threads load the entries coalesced, gather x and form
// each product and its rounding error into shared memory, and then one thread
// per row adds its row's terms in CSR order, so the sums keep the reference's
// order while loads and products run in parallel.
//
// The operator (rows, columns, values, L1 inverses, aggregates, members) does
// not change during a solve, so these kernels load their part of it before
// they wait for the previous kernel (griddepcontrol.wait): it was written at
// least one kernel before the predecessor, which itself started only after
// everything before it had completed. Vectors and the status are read after
// the wait only.
#include "common.cuh"
#include "kernels.hpp"

#include <algorithm>

namespace kb2 {
namespace {
using namespace dev;

// Adds entries [from, to) of the staged (product, error) pairs. For levels
// with long rows (kAhead > 0) the pairs of the next kAhead entries are loaded
// while the current ones are added: the chain is two dependent float additions
// per entry, and a shared-memory load in it would cost three times that.
template <int kAhead>
__device__ __forceinline__ void add_staged(float& sum, float& error, const float2* staged,
                                           int from, int to) {
  if constexpr (kAhead == 0) {
#pragma unroll 4
    for (; from < to; ++from) residual_add(sum, error, staged[from].x, staged[from].y);
  } else {
    float2 next[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) next[k] = staged[min(from + k, to - 1)];
    for (; from + kAhead < to; from += kAhead) {
      float2 now[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        now[k] = next[k];
        next[k] = staged[min(from + kAhead + k, to - 1)];
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) residual_add(sum, error, now[k].x, now[k].y);
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (from + k < to) residual_add(sum, error, next[k].x, next[k].y);
  }
}

enum class Rows { Residual, Smooth, SmoothProlonged };

// out = b - A x, or the sweep x + (2/3) inv (b - A x); SmoothProlonged reads
// x + coarse[aggregate] in the place of x (the prolongation, which adds it
// once per row, folded into the first post-sweep). kSorted: the block's rows go to
// its threads in the given order, longest first, so that a warp of short rows
// does not wait for a hub row in it.
template <int kRows, int kPer, int kAhead, Rows kMode, bool kSorted>
__global__ void __launch_bounds__(kBlock) k_staged_rows(
    int n, const int* __restrict__ rows, const int* __restrict__ cols,
    const float* __restrict__ vals, const float* __restrict__ inv, const float* __restrict__ x,
    const float* __restrict__ b, float* __restrict__ out, const int* __restrict__ status,
    const int* __restrict__ aggregate, const float* __restrict__ coarse,
    const int* __restrict__ order) {
  constexpr int kStage = kPer * kBlock;
  static_assert(kStage == launch::kStagedEntries * (kRows / launch::kStagedRows), "adds_too_long");
  constexpr bool kProlong = kMode == Rows::SmoothProlonged;
  __shared__ float2 staged[kStage];
  const int tid = threadIdx.x;
  const int row0 = blockIdx.x * kRows, row1 = min(n, row0 + kRows);
  const int first = rows[row0], last = rows[row1];
  const bool owner = tid < kRows && row0 + tid < n;
  const int i = kSorted && owner ? order[row0 + tid] : row0 + tid;
  const int begin = owner ? rows[i] : 0, end = owner ? rows[i + 1] : 0;
  const float scale = kMode != Rows::Residual && owner ? inv[i] : 0.0f;
  const int own_group = kProlong && owner ? aggregate[i] : -1;
  int c[kPer], g[kProlong ? kPer : 1];
  float v[kPer];
  const auto load = [&](int base) {
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int e = base + tid + k * kBlock;
      c[k] = e < last ? cols[e] : -1;
      v[k] = e < last ? vals[e] : 1.0f;
    }
    if constexpr (kProlong) {
#pragma unroll
      for (int k = 0; k < kPer; ++k) g[k] = c[k] >= 0 ? aggregate[c[k]] : -1;
    }
  };
  load(first);
  pdl_entry();
  const int stopped = status ? status[0] : 0;
  float sum = owner ? b[i] : 0.0f, error = 0.0f;
  float xi = kMode != Rows::Residual && owner ? x[i] : 0.0f;
  if (kProlong && own_group >= 0) xi += coarse[own_group];
  for (int base = first; base < last; base += kStage) {
    float xv[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      xv[k] = c[k] >= 0 ? x[c[k]] : 1.0f;
      if constexpr (kProlong)
        if (g[k] >= 0) xv[k] += coarse[g[k]];
    }
    // Work queued past the end of a solve stops here: after the gathers are
    // issued, so that the status adds no latency while the solve runs. (A solve
    // of 663,552 tets 14.9 ms against 15.4 with the status tested at the store only,
    // and 16.3 with it read before the operator's loads as well.)
    if (stopped != 0) return;
    float product[kPer], rounding[kPer];
    products(v, xv, product, rounding);
    if (base != first) __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (c[k] >= 0) staged[tid + k * kBlock] = make_float2(product[k], rounding[k]);
    __syncthreads();
    if (base + kStage < last) load(base + kStage);
    const int from = max(begin, base) - base, to = min(end, base + kStage) - base;
    if (from < to) add_staged<kAhead>(sum, error, staged, from, to);
  }
  if (stopped != 0 || !owner) return;
  out[i] = kMode != Rows::Residual ? xi + (2.0f / 3.0f) * scale * (sum + error) : sum + error;
}

// coarse = the Kahan sum over each aggregate's members (amg_restrict,
// src/kutta/kernels/amg.kern.h:5-16); with kZero also the coarse level's
// zero-start sweep of the row it just wrote (amg_smooth_zero). The members of
// an aggregate (8 or so) are loaded kBatch at a time, the first batch's
// indices before the wait.
template <bool kZero>
__global__ void __launch_bounds__(kBlock) k_restrict_rows(
    int nc, const int* __restrict__ offsets, const int* __restrict__ members,
    const float* __restrict__ fine, float* __restrict__ coarse, const int* __restrict__ rows,
    const float* __restrict__ vals, const float* __restrict__ inv, float* __restrict__ next,
    const int* __restrict__ status) {
  constexpr int kBatch = 8;
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const bool owner = g < nc;
  const int begin = owner ? offsets[g] : 0, end = owner ? offsets[g + 1] : 0;
  const float scale = kZero && owner ? inv[g] : 0.0f;
  int m[kBatch];
#pragma unroll
  for (int k = 0; k < kBatch; ++k) m[k] = begin + k < end ? members[begin + k] : -1;
  pdl_entry();
  const int stopped = status[0];
  float sum = 0.0f, error = 0.0f;
  for (int j = begin; j < end; j += kBatch) {
    float f[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) f[k] = m[k] >= 0 ? fine[m[k]] : 0.0f;
    if (stopped != 0) return;  // as in k_staged_rows
#pragma unroll
    for (int k = 0; k < kBatch; ++k)
      if (j + k < end) {
        const float term = f[k] - error;
        const float to = sum + term;
        error = (to - sum) - term;
        sum = to;
        m[k] = j + kBatch + k < end ? members[j + kBatch + k] : -1;
      }
  }
  if (stopped != 0 || !owner) return;
  coarse[g] = sum;
  if constexpr (kZero) next[g] = zero_sweep_row(g, rows, vals, sum, scale);
}

// ---- the small levels' V-cycle in one block ----------------------------------
//
// Levels of a few thousand entries cost a launch (1.5 us at best) per sweep,
// although a sweep of them is a microsecond of one SM's work; below
// kPlainTailRows rows the whole descent and ascent, the restriction into the
// first of them included, runs in one block of 1,024 threads with the level
// vectors and operators in shared memory; the operators are loaded before the
// wait for the previous kernel. One SM is bound by the instructions it issues,
// and a warp adds as long as its longest row. So rows go to threads in order
// of length, and the entries lie in slices of 32 rows with entry k of the
// slice's rows side by side (no bank conflicts), each with its column as a
// byte offset; once per refresh they are packed so. Levels of 512, 64 and 8
// rows under a V(5,5) cycle (59 passes) take 24 us, against 127 us as launches
// with the one-thread coarsest solve; levels of 1,439 and 854 rows (45
// passes, the longest row 56) 87 us against 105 us as launches of the kernels
// above and 350 us before them. No waits between blocks.
constexpr int kTailThreads = 1024;
constexpr int kTailRows = launch::kPlainTailRows / kTailThreads;  // rows of a thread

struct TailLevel {
  int row[kTailRows], start[kTailRows], length[kTailRows];
  float scale[kTailRows], right[kTailRows];
};

__device__ __forceinline__ void tail_load(const launch::PlainTail::Level& l, const float* b,
                                          TailLevel& t) {
#pragma unroll
  for (int q = 0; q < kTailRows; ++q) {
    const int at = threadIdx.x + q * kTailThreads;
    const bool owner = at < l.n;
    const int i = owner ? l.order[at] : -1;
    t.row[q] = i;
    t.start[q] = owner ? l.start[at] : 0;
    t.length[q] = owner ? l.rows[i + 1] - l.rows[i] : 0;
    t.scale[q] = owner ? l.inv[i] : 0.0f;
    t.right[q] = owner ? b[i] : 0.0f;
  }
}

__device__ __forceinline__ float tail_x(const float* x, float offset) {
  return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(x) +
                                         __float_as_int(offset));
}

// Adds a row's terms four at a time. The four errors take one check: every
// product at least 2^-96 and every factor at most 1e30 in magnitude (the
// minimum and maximum drop a NaN, whose error is NaN either way).
__device__ __forceinline__ void tail_add(float& sum, float& error, const float2* entry, int left,
                                         const float* x) {
  for (; left >= 4; left -= 4, entry += 4 * 32) {
    float2 e[4];
    float xv[4], product[4], rounding[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = entry[32 * k];
#pragma unroll
    for (int k = 0; k < 4; ++k) xv[k] = tail_x(x, e[k].y);
    float least = 1.0f, most = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      product[k] = e[k].x * xv[k];
      rounding[k] = fmaf(e[k].x, xv[k], -product[k]);
      least = fminf(least, fabsf(product[k]));
      most = fmaxf(most, fmaxf(fabsf(xv[k]), fabsf(e[k].x)));
    }
    if (!(least >= 0x1p-96f && most <= 1.0e30f)) {
#pragma unroll
      for (int k = 0; k < 4; ++k) rounding[k] = product_error_fma(e[k].x, xv[k], product[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) residual_add(sum, error, product[k], rounding[k]);
  }
  for (; left > 0; --left, entry += 32) residual_term(sum, error, entry->x, tail_x(x, entry->y));
}

// One pass over the level's rows: out = b - A x or the sweep from x.
template <bool kSmooth>
__device__ __forceinline__ void tail_rows(const TailLevel& t, const float2* entries,
                                          const float* x, float* out) {
#pragma unroll
  for (int q = 0; q < kTailRows; ++q)
    if (t.row[q] >= 0) {
      float sum = t.right[q], error = 0.0f;
      tail_add(sum, error, entries + t.start[q], t.length[q], x);
      const int i = t.row[q];
      out[i] = kSmooth ? x[i] + (2.0f / 3.0f) * t.scale[q] * (sum + error) : sum + error;
    }
  __syncthreads();
}

// Sweeps from x (or from zero) with y as the other buffer; returns the buffer
// that holds the result.
__device__ __forceinline__ float* tail_smooth(const launch::PlainTail::Level& l, const TailLevel& t,
                                              const float2* entries, float* x, float* y,
                                              int sweeps, bool zero) {
  for (int s = 0; s < sweeps; ++s) {
    if (zero && s == 0) {
#pragma unroll
      for (int q = 0; q < kTailRows; ++q)
        if (t.row[q] >= 0)
          x[t.row[q]] = zero_sweep_row(t.row[q], l.rows, l.vals, t.right[q], t.scale[q]);
      __syncthreads();
      continue;
    }
    tail_rows<true>(t, entries, x, y);
    float* swap = x;
    x = y;
    y = swap;
  }
  return x;
}

// The coarsest level's sweeps when it has at most 32 rows: one warp, a lane per
// row, no block barriers. The iterate ends in x.
__device__ __forceinline__ void tail_few_rows(const launch::PlainTail::Level& l,
                                              const float2* entries, float* x, const float* b,
                                              int sweeps) {
  if (threadIdx.x < 32) {
    TailLevel t;
    tail_load(l, b, t);
    const int i = t.row[0];
    if (i >= 0) x[i] = zero_sweep_row(i, l.rows, l.vals, t.right[0], t.scale[0]);
    __syncwarp();
    for (int s = 1; s < sweeps; ++s) {
      float sum = t.right[0], error = 0.0f;
      tail_add(sum, error, entries + t.start[0], t.length[0], x);
      const float next = i >= 0 ? x[i] + (2.0f / 3.0f) * t.scale[0] * (sum + error) : 0.0f;
      __syncwarp();
      if (i >= 0) x[i] = next;
      __syncwarp();
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void tail_restrict(const launch::PlainTail::Level& l, const float* fine,
                                              float* b) {
  for (int g = threadIdx.x; g < l.n; g += kTailThreads) {
    float sum = 0.0f, error = 0.0f;
    const int end = l.offsets[g + 1];
#pragma unroll 4
    for (int j = l.offsets[g]; j < end; ++j) {
      const float term = fine[l.members[j]] - error;
      const float next = sum + term;
      error = (next - sum) - term;
      sum = next;
    }
    b[g] = sum;
  }
  __syncthreads();
}

// The levels' entries in slices from their CSR values, once per refresh; all the
// levels' slots in one launch (2 us for each level otherwise).
__global__ void k_tail_entries(const __grid_constant__ launch::PlainTail t) {
  pdl_entry();
  const int at = blockIdx.x * blockDim.x + threadIdx.x;
  if (at >= t.slots) return;
  int k = t.levels - 1;
  while (at < t.level[k].slot) --k;
  const auto& l = t.level[k];
  const int e = l.source[at - l.slot];
  t.entries[at] =
      make_float2(e >= 0 ? l.vals[e] : 0.0f, __int_as_float(e >= 0 ? 4 * l.cols[e] : 0));
}

__global__ void __launch_bounds__(kTailThreads) k_plain_tail(const launch::PlainTail t,
                                                             const float* __restrict__ fine,
                                                             float* __restrict__ out,
                                                             const int* __restrict__ status) {
  extern __shared__ float2 tail_shared[];
  float* vectors = reinterpret_cast<float*>(tail_shared + t.slots);
  // The operators, 16 bytes a load, eight loads in flight.
  const float4* from = reinterpret_cast<const float4*>(t.entries);
  float4* to = reinterpret_cast<float4*>(tail_shared);
  for (int j = threadIdx.x; j < t.slots / 2; j += 8 * kTailThreads) {
    float4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j + k * kTailThreads < t.slots / 2) v[k] = from[j + k * kTailThreads];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (j + k * kTailThreads < t.slots / 2) to[j + k * kTailThreads] = v[k];
  }
  pdl_entry();
  if (status[0] != 0) return;
  __syncthreads();
  TailLevel now;
  const int last = t.levels - 1;
  // Where a level's iterate ends up in its two buffers: the zero-start sweep
  // writes the first, every other sweep moves to the other one. The residual
  // for the level below goes to the buffer that is free.
  const int down = (t.pre - 1) & 1, up = (down + t.post) & 1;
  const float* above = nullptr;
  for (int k = 0; k <= last; ++k) {
    const auto& l = t.level[k];
    const float2* entries = tail_shared + l.slot;
    float* x0 = vectors + l.at;
    float* b = x0 + 2 * l.n;
    if (k == 0)
      tail_restrict(l, fine, b);
    else
      tail_restrict(l, above, b);
    if (k == last && l.n <= 32) {
      tail_few_rows(l, entries, x0, b, t.coarsest);
      continue;
    }
    tail_load(l, b, now);
    float* x =
        tail_smooth(l, now, entries, x0, x0 + l.n, k < last ? t.pre : t.coarsest, true);
    if (k < last) {
      float* r = x == x0 ? x0 + l.n : x0;
      tail_rows<false>(now, entries, x, r);
      above = r;
    }
  }
  const int end = t.level[last].n <= 32 ? 0 : (t.coarsest - 1) & 1;
  const float* below = vectors + t.level[last].at + end * t.level[last].n;
  for (int k = last - 1; k >= 0; --k) {
    const auto& l = t.level[k];
    float* x0 = vectors + l.at;
    float* x = x0 + down * l.n;
    tail_load(l, x0 + 2 * l.n, now);
    for (int i = threadIdx.x; i < l.n; i += kTailThreads) {
      const int g = l.aggregate[i];
      if (g >= 0) x[i] += below[g];
    }
    __syncthreads();
    tail_smooth(l, now, tail_shared + l.slot, x, x0 + (down ^ 1) * l.n, t.post, false);
    below = x0 + up * l.n;
  }
  for (int i = threadIdx.x; i < t.level[0].n; i += kTailThreads) out[i] = below[i];
}

int row_blocks(int n, int rows) { return (n + rows - 1) / rows; }

template <Rows kMode>
void staged(int n, const int* rows, const int* cols, const float* vals, const float* inv,
            const float* x, const float* b, float* out, const int* status, const int* aggregate,
            const float* coarse, const int* order, cudaStream_t s) {
  ++launch::counter;
  // Few rows: 64 to a block, each thread one to four entries, with the adding
  // looked ahead (12,571 rows, longest 165: 3.8 us a sweep against 4.0 with the
  // larger form; 4,096 rows of up to 7: 2.0 against 2.1). More rows: 128 to a
  // block and plain adding, which leaves registers for more blocks (39,033 rows:
  // 3.6 us against 3.7; 48,848: 5.2 against 5.7; 159,785: 5.6 against 7.9).
  // An order comes with levels whose longest row has kStagedHub entries or more
  // (48,848 rows, longest 123: 4.4 us against 5.2; at 46 entries it gives nothing).
  if (n <= launch::kStagedSmall)
    pdl(k_staged_rows<64, 4, 4, kMode, false>, row_blocks(n, 64), kBlock, 0, s, n, rows, cols,
        vals, inv, x, b, out, status, aggregate, coarse, order);
  else if (order != nullptr)
    pdl(k_staged_rows<128, 8, 0, kMode, true>, row_blocks(n, 128), kBlock, 0, s, n, rows, cols,
        vals, inv, x, b, out, status, aggregate, coarse, order);
  else
    pdl(k_staged_rows<128, 8, 0, kMode, false>, row_blocks(n, 128), kBlock, 0, s, n, rows, cols,
        vals, inv, x, b, out, status, aggregate, coarse, order);
}

}  // namespace

namespace launch {

void staged_residual(int n, const int* rows, const int* cols, const float* vals, const float* x,
                     const float* b, float* r, const int* status, const int* order,
                     cudaStream_t s) {
  if (n <= 0) return;
  staged<Rows::Residual>(n, rows, cols, vals, nullptr, x, b, r, status, nullptr, nullptr, order,
                         s);
}

void staged_smooth(int n, const int* rows, const int* cols, const float* vals, const float* x,
                   const float* b, const float* inv, float* next, const int* status,
                   const int* aggregate, const float* coarse, const int* order, cudaStream_t s) {
  if (n <= 0) return;
  if (aggregate != nullptr)
    staged<Rows::SmoothProlonged>(n, rows, cols, vals, inv, x, b, next, status, aggregate, coarse,
                                  order, s);
  else
    staged<Rows::Smooth>(n, rows, cols, vals, inv, x, b, next, status, nullptr, nullptr, order, s);
}

void restrict_rows(int nc, const int* offsets, const int* members, const float* fine,
                   float* coarse, const int* rows, const float* vals, const float* inv,
                   float* next, const int* status, cudaStream_t s) {
  if (nc <= 0) return;
  ++counter;
  if (next != nullptr)
    pdl(k_restrict_rows<true>, row_blocks(nc, kBlock), kBlock, 0, s, nc, offsets, members, fine,
        coarse, rows, vals, inv, next, status);
  else
    pdl(k_restrict_rows<false>, row_blocks(nc, kBlock), kBlock, 0, s, nc, offsets, members, fine,
        coarse, rows, vals, inv, next, status);
}

int plain_tail_bytes(int floats, int slots) {
  return floats * static_cast<int>(sizeof(float)) + slots * static_cast<int>(sizeof(float2));
}

void plain_tail_entries(const PlainTail& t, cudaStream_t s) {
  if (t.slots <= 0) return;
  ++counter;
  pdl(k_tail_entries, row_blocks(t.slots, kBlock), kBlock, 0, s, t);
}

void plain_tail(const PlainTail& t, const float* fine, float* out, const int* status,
                cudaStream_t s) {
  static std::atomic<unsigned long long> raised{0};
  raise_shared_limit(reinterpret_cast<const void*>(k_plain_tail), kPlainTailBytes, raised);
  ++counter;
  pdl(k_plain_tail, 1, kTailThreads, plain_tail_bytes(t.floats, t.slots), s, t, fine, out, status);
}

}  // namespace launch
}  // namespace kb2
