// The finite-volume steps on either side of the pressure solve
// (src/kutta/kernels/fv_flow.kern.h:164-201), compiled without FMA
// contraction so every value rounds as the reference's CPU kernels do:
//
//   fv_pressure_assemble  cell i's CSR row of the pressure-correction matrix
//                         and its right-hand side from the face coefficients
//                         and mass fluxes (:164-183); with `fused`, the row's
//                         inverse L1 diagonal (the refresh's first step,
//                         linalg.kern.h:52-70) and its validity flag, the row's
//                         surplus for the level below and its packed copy follow
//                         in the same pass;
//   fv_correct_flux       face flux correction (:185-190);
//   fv_correct_velocity   cell velocity and pressure correction (:192-201).
//
// Row i's values are written only by the thread of row i (the entries of its
// faces and its diagonal are all in row i), so rows are independent.
#include <cuda_runtime.h>

#include "common.cuh"
#include "epilogues.cuh"
#include "kernels.hpp"

namespace kb2 {
namespace {
using namespace dev;

#define ROWS(i, n) \
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

struct Assembly {
  const int* offsets;
  const int* faces;
  const float* sign;
  const int* adjacent;
  const int* entry;
  const int* rows;
  const int* diag;
  const float* coefficient;
  const float* flux;
  int reference;
};

// Faces of a cell whose loads are issued together.
constexpr int kFaces = 4;

// Row i's values into `values`; returns its right-hand side. Bound by the loads'
// latency, the more so as the registers of register_row leave five blocks on an SM:
// one face after another, 1,000,000 rows took 266 us (11 entries on average) and
// 342 (13) in a kernel of its own, 294 and 368 beside register_row, and 227 and 280
// with four faces' loads issued together.
__device__ __forceinline__ float assemble_row(int i, const Assembly& a,
                                              float* __restrict__ values) {
  UpperSum ap{0.0f, 0.0f};
  float b = 0.0f;
  const int begin = __ldg(a.offsets + i), end = __ldg(a.offsets + i + 1);
  for (int first = begin; first < end; first += kFaces) {
    int entry[kFaces];
#pragma unroll
    for (int u = 0; u < kFaces; ++u)
      entry[u] = first + u < end && __ldg(a.adjacent + first + u) >= 0
                     ? __ldg(a.entry + first + u)
                     : -1;
#pragma unroll
    for (int u = 0; u < kFaces; ++u)
      if (entry[u] >= 0) values[entry[u]] = 0.0f;
  }
  for (int first = begin; first < end; first += kFaces) {
    int face[kFaces], nb[kFaces], entry[kFaces];
    float sign[kFaces], d[kFaces], flux[kFaces];
#pragma unroll
    for (int u = 0; u < kFaces; ++u) {
      const bool in = first + u < end;
      face[u] = in ? __ldg(a.faces + first + u) : -1;
      nb[u] = in ? __ldg(a.adjacent + first + u) : -1;
      entry[u] = in ? __ldg(a.entry + first + u) : -1;
      sign[u] = in ? __ldg(a.sign + first + u) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kFaces; ++u) {
      d[u] = face[u] >= 0 ? __ldg(a.coefficient + face[u]) : 0.0f;
      flux[u] = face[u] >= 0 ? __ldg(a.flux + face[u]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kFaces; ++u) {
      if (face[u] < 0) continue;
      b -= sign[u] * flux[u];
      // Boundary faces and the eliminated reference cell anchor the diagonal.
      if (nb[u] < 0 || nb[u] == a.reference) ap = upper_add(ap, d[u]);
      if (nb[u] >= 0 && nb[u] != a.reference && i != a.reference) values[entry[u]] -= d[u];
    }
  }
  // The stored off-diagonals once each (faces may share an entry), upward
  // rounded: the row stays weakly diagonally dominant.
  const int at = a.diag[i];
  row_values(values, a.rows[i], a.rows[i + 1], [&](int j, float v) {
    if (j != at) ap = upper_add(ap, -v);
  });
  values[at] = i == a.reference ? 1.0f : upper_value(ap);
  return i == a.reference ? 0.0f : b;
}

// A row of at most kRow off-diagonals (tetrahedra have four, hexahedra six) held
// in registers: its faces are taken kFaces at a time, their loads issued together
// and then the gathers, and each is added to the off-diagonal that its entry
// names instead of in memory; an entry that no face has keeps the value that it
// had. Sums and their order are assemble_row's, and those of diagonal_row,
// row_surplus and pack_row. Five dependent passes over the row in memory took
// 127 us at 1,572,864 tetrahedra with the fused parts, this 72, for 220 MB that
// have to move. (Rows of at most six faces only: 117, as one cell in twenty there
// has more and its warp then runs both forms.)
constexpr int kRow = 6;
template <bool kFused>
__device__ __forceinline__ float register_row(int i, int begin, int count, int at,
                                              const Assembly& a, float* __restrict__ values,
                                              float* __restrict__ rhs,
                                              const launch::FvFused& fused) {
  float v[kRow];
  unsigned found = 0;
  UpperSum ap{0.0f, 0.0f};
  float b = 0.0f;
#pragma unroll
  for (int k = 0; k < kRow; ++k) v[k] = 0.0f;
  const int end = __ldg(a.offsets + i + 1);
  for (int first = __ldg(a.offsets + i); first < end; first += kFaces) {
    int face[kFaces], nb[kFaces], entry[kFaces];
    float sign[kFaces], d[kFaces], flux[kFaces];
#pragma unroll
    for (int u = 0; u < kFaces; ++u) {
      const bool in = first + u < end;
      face[u] = in ? __ldg(a.faces + first + u) : -1;
      nb[u] = in ? __ldg(a.adjacent + first + u) : -1;
      entry[u] = in ? __ldg(a.entry + first + u) : -1;
      sign[u] = in ? __ldg(a.sign + first + u) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kFaces; ++u) {
      d[u] = face[u] >= 0 ? __ldg(a.coefficient + face[u]) : 0.0f;
      flux[u] = face[u] >= 0 ? __ldg(a.flux + face[u]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kFaces; ++u) {
      if (face[u] < 0) continue;
      b -= sign[u] * flux[u];
      if (nb[u] < 0 || nb[u] == a.reference) ap = upper_add(ap, d[u]);
      // (A face between a cell and itself names the diagonal, which is set last.)
      if (nb[u] < 0 || entry[u] == at) continue;
      const int slot = entry[u] - begin - (entry[u] > at);
      found |= 1u << slot;
      const int into = nb[u] != a.reference && i != a.reference ? slot : -1;
#pragma unroll
      for (int k = 0; k < kRow; ++k)
        if (into == k) v[k] -= d[u];
    }
  }
#pragma unroll
  for (int k = 0; k < kRow; ++k) {
    if (k >= count) continue;
    const int j = begin + k + (begin + k >= at);
    if (found >> k & 1u)
      values[j] = v[k];
    else
      v[k] = values[j];
    ap = upper_add(ap, -v[k]);
  }
  const float centre = i == a.reference ? 1.0f : upper_value(ap);
  values[at] = centre;
  rhs[i] = i == a.reference ? 0.0f : b;
  if constexpr (!kFused) return 0.0f;
  float off = 0.0f, bad = centre - centre != 0.0f ? 1.0f : 0.0f;
  UpperSum sum{centre, 0.0f};
#pragma unroll
  for (int k = 0; k < kRow; ++k) {
    if (k >= count) continue;
    if (v[k] - v[k] != 0.0f) bad = 1.0f;
    off += fabsf(v[k]);
    sum = upper_add(sum, v[k]);
  }
  if (fused.surplus != nullptr) fused.surplus[i] = upper_value(sum);
  if (fused.width > 0) {
    // Packed rows are 4 or 8 wide; a wider row than the width is not packed.
    float4* out = reinterpret_cast<float4*>(fused.packed + static_cast<std::size_t>(i) * fused.width);
    const auto value = [&](int k) { return k < kRow && k < count ? v[k < kRow ? k : 0] : 0.0f; };
    out[0] = make_float4(value(0), value(1), value(2), value(3));
    if (fused.width > 4) out[1] = make_float4(value(4), value(5), value(6), value(7));
    fused.packed_diag[i] = centre;
  }
  return diagonal_value(centre, off, bad, 1, fused.inverse[i]);
}

template <bool kFused>
__global__ void __launch_bounds__(kBlock, 5)
    k_fv_pressure_assemble(int n, Assembly a, float* __restrict__ values, float* __restrict__ rhs,
                           launch::FvFused fused, DeviceReducer red, double* check, int slot) {
  pdl_entry();
  double worst = 0;
  ROWS(i, n) {
    const int begin = __ldg(a.rows + i), count = __ldg(a.rows + i + 1) - begin - 1;
    const int at = __ldg(a.diag + i);
    if (count <= kRow) {
      const float flag = register_row<kFused>(i, begin, count, at, a, values, rhs, fused);
      if constexpr (kFused) worst = nan_max(worst, flag);
      continue;
    }
    rhs[i] = assemble_row(i, a, values);
    if constexpr (kFused) {
      worst = nan_max(worst, diagonal_row(i, a.rows, a.diag, values, fused.inverse, 1));
      if (fused.surplus != nullptr) fused.surplus[i] = row_surplus(i, a.rows, a.diag, values);
      if (fused.width > 0)
        pack_row(i, fused.width, a.rows, a.diag, values, fused.packed, fused.packed_diag);
    }
  }
  if constexpr (kFused) finish_max(as_reducer(red), worst, check, slot);
}

__global__ void k_fv_correct_flux(int n, const int* __restrict__ owner,
                                  const int* __restrict__ neighbour,
                                  const float* __restrict__ correction,
                                  const float* __restrict__ coefficient, float* __restrict__ flux,
                                  int internal) {
  pdl_entry();
  ROWS(i, n) {
    const float pc = correction[owner[i]];
    const float pn = i < internal ? correction[neighbour[i]] : 0.0f;
    flux[i] += coefficient[i] * (pc - pn);
  }
}

__global__ void k_fv_correct_velocity(int n, const float* __restrict__ volume,
                                      const float* __restrict__ inverse,
                                      const float* __restrict__ diagonal,
                                      const float* __restrict__ gx, const float* __restrict__ gy,
                                      const float* __restrict__ gz,
                                      const float* __restrict__ correction, float* __restrict__ u,
                                      float* __restrict__ v, float* __restrict__ w,
                                      float* __restrict__ p, float alpha) {
  pdl_entry();
  ROWS(i, n) {
    const float d = volume[i] * inverse[i];
    u[i] -= d * gx[i];
    v[i] -= d * gy[i];
    w[i] -= d * gz[i];
    // The pressure step is bounded by the local ratio of the physical to the
    // SIMPLEC correction coefficient.
    const float pressure_alpha = fminf(alpha, 0.7f * diagonal[i] * inverse[i]);
    p[i] += pressure_alpha * correction[i];
  }
}

}  // namespace

namespace launch {

void fv_pressure_assemble(int n, const int* offsets, const int* faces, const float* sign,
                          const int* adjacent, const int* entry, const int* rows, const int* diag,
                          const float* coefficient, const float* flux, float* values, float* rhs,
                          int reference, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  const Assembly a{offsets, faces, sign, adjacent, entry, rows, diag, coefficient, flux, reference};
  pdl(k_fv_pressure_assemble<false>, grid_for(n), kBlock, 0, s, n, a, values, rhs, FvFused{},
      DeviceReducer{nullptr, nullptr}, static_cast<double*>(nullptr), 0);
}

void fv_pressure_assemble_l1(int n, const int* offsets, const int* faces, const float* sign,
                             const int* adjacent, const int* entry, const int* rows,
                             const int* diag, const float* coefficient, const float* flux,
                             float* values, float* rhs, int reference, const FvFused& fused,
                             DeviceReducer red, double* check, int slot, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  const Assembly a{offsets, faces, sign, adjacent, entry, rows, diag, coefficient, flux, reference};
  pdl(k_fv_pressure_assemble<true>, grid_for(n), kBlock, 0, s, n, a, values, rhs, fused, red, check,
      slot);
}

void fv_correct_flux(int n, const int* owner, const int* neighbour, const float* correction,
                     const float* coefficient, float* flux, int internal, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_fv_correct_flux, grid_for(n), kBlock, 0, s, n, owner, neighbour, correction, coefficient,
      flux, internal);
}

void fv_correct_velocity(int n, const float* volume, const float* inverse, const float* diagonal,
                         const float* gx, const float* gy, const float* gz,
                         const float* correction, float* u, float* v, float* w, float* p,
                         float alpha, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_fv_correct_velocity, grid_for(n), kBlock, 0, s, n, volume, inverse, diagonal, gx, gy, gz,
      correction, u, v, w, p, alpha);
}

}  // namespace launch
}  // namespace kb2
