// The mixed solve's smallest levels in one block (no reference counterpart).
//
// Levels of up to a thousand rows and the dense coarsest below them cost a few
// microseconds of launch and memory latency per step, whatever the step does: at
// 859 and 107 rows two inner Krylov steps were 20 launches and 26 us, this kernel
// 11. One block of 1,024 threads, a thread per row, holds the operators, the
// transfers, the dense inverse and every vector in shared memory. It is bound by
// instructions and barriers, so a sweep's inner loop is one word per entry (BF16
// value and the column's byte offset) from slices of 32 rows in order of length,
// five instructions an entry; four lanes per row over the CSR rows, as the larger
// levels' kernels have them, took 18 us for what takes 11 here. The image that is
// loaded is laid out with the hierarchy and its values are set by each refresh,
// which the host waits for, so that it is loaded before the wait for the previous
// kernel. Row sums keep the order of the separate kernels (four partial sums).
#include <atomic>

#include "common.cuh"
#include "inner_steps.cuh"
#include "kernels.hpp"

namespace kb2 {
namespace {
using namespace dev;
using launch::MixedTail;
using Level = MixedTail::Level;

constexpr int kThreads = MixedTail::kMaxRows;
constexpr float kOmega = 2.0f / 3.0f;

template <typename T>
__device__ __forceinline__ T* shared_at(float* shared, int at) {
  return reinterpret_cast<T*>(shared + at);
}
__device__ __forceinline__ float at_byte(const float* x, unsigned offset) {
  return *reinterpret_cast<const float*>(reinterpret_cast<const char*>(x) + offset);
}

// The thread's sum over its slice's slots, four partial sums as four lanes keep
// them; term(word) for each. A slice's slots are padded to a multiple of four with
// words that add a zero.
template <class Term>
__device__ __forceinline__ float slice_sum(float* shared, int slices_at, int slots_at, Term term) {
  const int2 slice = shared_at<int2>(shared, slices_at)[threadIdx.x >> 5];
  const unsigned* slot = shared_at<unsigned>(shared, slots_at) + slice.x + (threadIdx.x & 31);
  float acc[4] = {};
  for (int j = 0; j < slice.y; j += 4) {
    unsigned word[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) word[u] = slot[32 * (j + u)];
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = term(acc[u], word[u]);
  }
  return (acc[0] + acc[2]) + (acc[1] + acc[3]);
}

// sum_j a_ij x_j / scale_i of row i = threadIdx.x (for all threads of a warp with a row).
__device__ __forceinline__ float product(float* shared, const Level& l, const float* x) {
  return slice_sum(shared, l.slices_at, l.entries_at, [&](float acc, unsigned e) {
    return fmaf(__uint_as_float(e & 0xffff0000u), at_byte(x, e & 0xffffu), acc);
  });
}

// One V-cycle over the tail; `top` is the first level's right-hand side at the
// thread's row. The iterate ends in buffer (pre + post) of the first level.
// After k sweeps a level's iterate is in its first buffer if k is odd.
__device__ __forceinline__ float* buffer(float* shared, const Level& l, int sweeps) {
  return shared + (sweeps & 1 ? l.x_at : l.r_at);
}
__device__ float* v_cycle(float* shared, const MixedTail& t, float top) {
  const int last = t.levels - 1, i = threadIdx.x;
  if (i < t.level[0].n)
    buffer(shared, t.level[0], 1)[i] = kOmega * shared[t.level[0].inv_at + i] * top;
  __syncthreads();
  for (int k = 0; k < last; ++k) {
    const Level& l = t.level[k];
    const Level& c = t.level[k + 1];
    const bool mine = i < l.n;
    const float right = mine ? (k == 0 ? top : shared[l.b_at + i]) : 0.0f;
    const float scale = mine ? shared[l.scale_at + i] : 0.0f;
    const float inv = mine ? shared[l.inv_at + i] : 0.0f;
    for (int s = 1; s < t.pre; ++s) {
      const float* x = buffer(shared, l, s);
      if (mine)
        buffer(shared, l, s + 1)[i] =
            x[i] + kOmega * inv * (right - scale * product(shared, l, x));
      __syncthreads();
    }
    float* r = buffer(shared, l, t.pre + 1);
    if (mine) r[i] = right - scale * product(shared, l, buffer(shared, l, t.pre));
    __syncthreads();
    if (i < c.n) {
      const float sum = slice_sum(shared, l.groups_at, l.members_at,
                                  [&](float acc, unsigned e) { return acc + at_byte(r, e); });
      if (k + 1 < last) {
        shared[c.b_at + i] = sum;
        buffer(shared, c, 1)[i] = kOmega * shared[c.inv_at + i] * sum;
      } else {
        shared_at<double>(shared, c.b_at)[i] = static_cast<double>(sum);
      }
    }
    if (k + 1 == last) asm volatile("cp.async.wait_all;" ::: "memory");  // the inverse
    __syncthreads();
  }
  {
    // The coarsest: eight lanes per row of the inverse.
    const Level& l = t.level[last];
    const double* inverse = shared_at<double>(shared, l.entries_at);
    const double* right = shared_at<double>(shared, l.b_at);
    const int lane = i & 7;
    for (int row0 = (i >> 5) * 4; row0 < l.n; row0 += kThreads / 8) {
      const int row = row0 + ((i & 31) >> 3);
      double acc = 0.0;
      if (row < l.n) {
#pragma unroll 4
        for (int k = lane; k < l.n; k += 8) acc += inverse[row * l.n + k] * right[k];
      }
      for (int d = 4; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d, 8);
      if (row < l.n && lane == 0) shared[l.x_at + row] = static_cast<float>(acc);
    }
    __syncthreads();
  }
  const float* coarse = shared + t.level[last].x_at;
  for (int k = last - 1; k >= 0; --k) {
    const Level& l = t.level[k];
    const bool mine = i < l.n;
    if (mine) {
      const int g = shared_at<int>(shared, l.aggregate_at)[i];
      if (g >= 0) buffer(shared, l, t.pre)[i] += coarse[g];
    }
    const float right = mine ? (k == 0 ? top : shared[l.b_at + i]) : 0.0f;
    const float scale = mine ? shared[l.scale_at + i] : 0.0f;
    const float inv = mine ? shared[l.inv_at + i] : 0.0f;
    __syncthreads();
    for (int s = t.pre; s < t.pre + t.post; ++s) {
      const float* x = buffer(shared, l, s);
      if (mine)
        buffer(shared, l, s + 1)[i] =
            x[i] + kOmega * inv * (right - scale * product(shared, l, x));
      __syncthreads();
    }
    coarse = buffer(shared, l, t.pre + t.post);
  }
  return buffer(shared, t.level[0], t.pre + t.post);
}

// The block's totals of a and b as pairs at scalars[at], scalars[at + 2], then
// step() in one thread; scalars and what step() writes are shared memory.
template <class Step>
__device__ __forceinline__ void total2(double a, double b, float* scalars, int at, Step step) {
  __shared__ double sums[64];
  a = warp_sum(a);
  b = warp_sum(b);
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    sums[warp] = a;
    sums[32 + warp] = b;
  }
  __syncthreads();
  if (warp == 0) {
    a = warp_sum(sums[threadIdx.x]);
    b = warp_sum(sums[32 + threadIdx.x]);
    if (threadIdx.x == 0) {
      store_pair(scalars, at, a);
      store_pair(scalars, at + 2, b);
      step();
    }
  }
  __syncthreads();
}

// q = A p at the thread's row, then p.q and w.p -> scalars[0..3] and the step length.
__device__ __forceinline__ float product_step(float* shared, const Level& l, const float* p,
                                              float w, float* scalars, int* status, bool first) {
  const int i = threadIdx.x;
  double a = 0.0, b = 0.0;
  float q = 0.0f;
  if (i < l.n) {
    q = shared[l.scale_at + i] * product(shared, l, p);
    a = static_cast<double>(p[i]) * static_cast<double>(q);
    b = static_cast<double>(w) * static_cast<double>(p[i]);
  }
  total2(a, b, scalars, 0, [&] { inner_alpha(scalars, status, first); });
  return q;
}

// out = the V-cycle's correction for the right-hand side `rhs`, or with kInner
// that of the two inner Krylov steps (Solver::inner) on the first tail level.
template <bool kInner>
__global__ void __launch_bounds__(kThreads)
    k_mixed_tail(const __grid_constant__ MixedTail t, const float* __restrict__ rhs,
                 float* __restrict__ out, const int* __restrict__ parent) {
  extern __shared__ __align__(16) float shared[];
  const unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(shared));
  const char* image = reinterpret_cast<const char*>(t.image);
  const auto fetch = [&](int from, int to) {  // words, multiples of 4
    for (int k = from / 4 + static_cast<int>(threadIdx.x); k < to / 4; k += kThreads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + 16 * k),
                   "l"(image + 16 * k)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, t.inverse_at);
  fetch(t.inverse_at, t.image_words);
  // The entry after each gathered vector is what padding words read.
  for (int k = threadIdx.x; k < t.levels - 1; k += kThreads)
    shared[t.level[k].x_at + t.level[k].n] = shared[t.level[k].r_at + t.level[k].n] = 0.0f;
  const Level& top = t.level[0];
  const int i = threadIdx.x;
  float* p = shared + t.p_at;
  if (kInner && i == 0) p[top.n] = 0.0f;
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  const bool mine = i < top.n;
  const int at = mine ? shared_at<int>(shared, t.order_at)[i] : 0;
  pdl_entry();
  if (parent[0] != 0) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  const float b = mine ? rhs[at] : 0.0f;
  float* z = v_cycle(shared, t, b);
  if constexpr (!kInner) {
    if (mine) out[at] = z[i];
    return;
  }
  __shared__ float scalars[16];
  __shared__ int status[1];
  if (i == 0) status[0] = 0;
  if (mine) p[i] = z[i];
  __syncthreads();
  const float q = product_step(shared, top, p, b, scalars, status, true);
  const bool running = status[0] == 0;
  const float first = running ? kp_float(kp_load(scalars, 8)) : 0.0f;
  const float r = running && mine ? b - first * q : 0.0f;
  float x = !mine ? 0.0f : (running ? first * p[i] : p[i]);
  if (running) {
    total2(static_cast<double>(r) * static_cast<double>(r),
           static_cast<double>(b) * static_cast<double>(b), scalars, 4,
           [&] { inner_check(scalars, status); });
    if (status[0] == 0) {
      z = v_cycle(shared, t, r);
      total2(mine ? static_cast<double>(z[i]) * static_cast<double>(q) : 0.0, 0.0, scalars, 4,
             [&] { inner_beta(scalars, status); });
    }
    if (status[0] == 0) {
      const float beta = kp_float(kp_load(scalars, 10));
      if (mine) p[i] = __fadd_rn(z[i], __fmul_rn(beta, p[i]));
      __syncthreads();
      product_step(shared, top, p, r, scalars, status, false);
    }
    if (status[0] == 0) {
      const float alpha = kp_float(kp_load(scalars, 8));
      if (mine) x = __fadd_rn(x, __fmul_rn(alpha, p[i]));
    }
  }
  if (mine) out[at] = x;
}

// A level's values into the image: each slot's BF16 value beside its column, the
// rows' scale and inverse diagonal in the image's order.
__global__ void k_mixed_tail_values(MixedTail::Values v, unsigned* __restrict__ image) {
  pdl_entry();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < v.slots) {
    const int e = v.source[k];
    unsigned* word = image + v.entries_at + k;
    if (e >= 0) *word = (v.packed[e] & 0xffff0000u) | (*word & 0xffffu);
  }
  if (k < v.n) {
    const int i = v.order[k];
    image[v.scale_at + k] = __float_as_uint(v.scale[i]);
    image[v.inv_at + k] = __float_as_uint(v.inv[i]);
  }
}

}  // namespace

namespace launch {

void mixed_tail_values(const MixedTail::Values& v, unsigned* image, cudaStream_t s) {
  ++counter;
  const int most = v.slots > v.n ? v.slots : v.n;
  pdl(k_mixed_tail_values, (most + kBlock - 1) / kBlock, kBlock, 0, s, v, image);
}

void mixed_tail(const MixedTail& t, const float* right, float* out, const int* status,
                cudaStream_t s) {
  static std::atomic<unsigned long long> raised[2] = {};
  ++counter;
  if (t.inner) {
    raise_shared_limit(reinterpret_cast<const void*>(k_mixed_tail<true>), MixedTail::kMaxBytes,
                       raised[1]);
    pdl(k_mixed_tail<true>, 1, kThreads, t.bytes, s, t, right, out, status);
  } else {
    raise_shared_limit(reinterpret_cast<const void*>(k_mixed_tail<false>), MixedTail::kMaxBytes,
                       raised[0]);
    pdl(k_mixed_tail<false>, 1, kThreads, t.bytes, s, t, right, out, status);
  }
}

}  // namespace launch
}  // namespace kb2
