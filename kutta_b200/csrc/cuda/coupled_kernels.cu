// Coupled (4x4-block) pressure-velocity solve kernels for sm_100a (compiled
// with --fmad=false, IEEE division): the block Jacobian of momentum and
// continuity in cell unknowns (u, v, w, p~), its damped block-Jacobi smoother,
// the piecewise-constant aggregation Galerkin operators and the transfers of
// src/kutta/kernels/fv_coupled.kern.h. Every per-row and per-coarse-row result
// rounds exactly as the reference kernel's: the same operations in the same
// order, no contraction.
//
// Layout on the device (own design; the reference keeps 4n planes, a 27n
// packed cell array and five incidence planes):
// - block vectors are float4 per cell (u, v, w, p~): one 16-byte load per
//   cell and per neighbour in the row kernels instead of four gathers;
// - setup-time cell data keeps the reference's 27 planes of n floats
//   (slot k of cell i at k n + i: du dv dw cd | Gx Gy Gz | Hx Hy Hz | Q (9) | cs
//   | 7 free), because the assembly kernels fill them slot by slot and the
//   fine Galerkin reads them;
// - the fine operator used every iteration is repacked once per solve into
//   per-cell records, 16-byte aligned: (du, dv, dw, cd), (wc Gx, wc Gy, wc Gz,
//   wc Hx), (wc Hy, wc Hz) and the block inverse's Schur denominator, and ELL
//   slots in slot-major order for the internal faces of each cell in cell-face order: (a, gx, gy,
//   gz), h and (neighbour, face) per slot, plus one (sx, sy, sz, rc) record
//   per face. A warp's slot loads are then contiguous 512-byte lines;
// - coarse levels (coupled_coarse.cu) keep the reference's CSR pattern with one
//   32-byte record per entry, (a, gx, gy, gz), (c, hx, hy, hz), and 11 planes of
//   n per row (du dv dw cs iu iv iw hx iu hy iv hz iw schur).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "coupled_kernels.hpp"
#include "coupled_rows.cuh"
#include "epilogues.cuh"

namespace kb2 {
namespace {

using namespace dev;

// Cell c's share of the face velocity it shares with cell i
// (fv_coupled.kern.h:86-91).
__device__ __forceinline__ float share_of(const float* __restrict__ weight, int i, int c) {
  return weight[c] / fmaxf(weight[i] + weight[c], 1.0e-30f);
}

// ---- Jacobian assembly, once per solve --------------------------------------

// fv_coupled.kern.h:183-189 (coupled_copy_diagonal).
__global__ void k_cpl_copy_diagonal(int n, const int* __restrict__ rows,
                                    const int* __restrict__ diag, const float* __restrict__ values,
                                    const float* __restrict__ physical, float* __restrict__ plane,
                                    float inverse_courant) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int d = diag[i];
    float off = 0.0f;
    for (int j = rows[i]; j < rows[i + 1]; ++j)
      if (j != d) off += fabsf(values[j]);
    const float p = physical[i];
    const float floored = fmaxf(p, off);
    plane[i] = values[d] + (floored - p) + inverse_courant * floored;
  }
}

// fv_coupled.kern.h:112-126 (coupled_face_coefficient), one thread per face.
__global__ void k_cpl_face_coefficient(int nf, int internal, const int* __restrict__ owner,
                                       const int* __restrict__ neighbour,
                                       const int* __restrict__ kind,
                                       const float* __restrict__ diffusion,
                                       const float* __restrict__ volume,
                                       const float* __restrict__ diagonal,
                                       float* __restrict__ coefficient, float scale) {
  pdl_entry();
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    const int c = owner[f];
    float rc = volume[c] / fmaxf(diagonal[c], 1.0e-20f);
    if (f < internal) {
      const int m = neighbour[f];
      rc = 0.5f * (rc + volume[m] / fmaxf(diagonal[m], 1.0e-20f));
    } else {
      const int k = kind[f - internal];
      if (k != 2 && k != 4) {
        coefficient[f] = 0.0f;
        continue;
      }
    }
    coefficient[f] = scale * rc * diffusion[f];
  }
}

struct FineGeometry {
  const int* offsets;
  const int* faces;
  const float* sign;
  const int* adjacent;
  const float *sx, *sy, *sz;
  const float *dx, *dy, *dz;
};

// One pass over each cell's faces for three of the reference's kernels, whose
// sums are independent (each in its own order): coupled_velocity_block
// (fv_coupled.kern.h:93-108), H_ii into planes 7-9; coupled_rhs (:131-150), the
// pressure diagonal into plane 3 and the block right-hand side; and
// coupled_fine_gsum (:191-208), the |G| row sums, 3n planes. Bound by the face
// data's latency: as three kernels 130 us at 884,736 hexes, this 75.
__global__ void __launch_bounds__(kBlock, 5) k_cpl_cell_sums(
    int n, int internal, FineGeometry m, const int* __restrict__ kind,
    const float* __restrict__ weight, const float* __restrict__ coefficient,
    const float* __restrict__ mass, const float* __restrict__ net, const float* __restrict__ ru,
    const float* __restrict__ rv, const float* __restrict__ rw, float* __restrict__ cell,
    float* __restrict__ r, float4* __restrict__ b, int reference, float continuity_scale,
    float wc) {
  pdl_entry();
  const std::size_t N = n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float q00 = wc * cell[10 * N + i], q01 = wc * cell[11 * N + i], q02 = wc * cell[12 * N + i];
    const float q10 = wc * cell[13 * N + i], q11 = wc * cell[14 * N + i], q12 = wc * cell[15 * N + i];
    const float q20 = wc * cell[16 * N + i], q21 = wc * cell[17 * N + i], q22 = wc * cell[18 * N + i];
    const float half_wc = 0.5f * wc;
    float gx = fabsf(wc * cell[4 * N + i]), gy = fabsf(wc * cell[5 * N + i]),
          gz = fabsf(wc * cell[6 * N + i]);
    float hx = 0.0f, hy = 0.0f, hz = 0.0f;
    Csum c{0.0f, 0.0f};
    float imbalance = 0.0f;
    for (int j = m.offsets[i]; j < m.offsets[i + 1]; ++j) {
      const int f = m.faces[j], other = m.adjacent[j];
      const float s = m.sign[j], sx = m.sx[f], sy = m.sy[f], sz = m.sz[f];
      c = csum_add(c, coefficient[f]);
      imbalance += s * mass[f];
      float share = 0.0f;
      if (other >= 0) {
        share = 1.0f - share_of(weight, i, other);
        gx += fabsf(half_wc * s * sx + q00 * m.dx[j] + q01 * m.dy[j] + q02 * m.dz[j]);
        gy += fabsf(half_wc * s * sy + q10 * m.dx[j] + q11 * m.dy[j] + q12 * m.dz[j]);
        gz += fabsf(half_wc * s * sz + q20 * m.dx[j] + q21 * m.dy[j] + q22 * m.dz[j]);
      } else {
        const int k = kind[f - internal];
        if (k == 2 || k == 4) share = 1.0f;
      }
      const float t = share * s;
      hx += t * sx;
      hy += t * sy;
      hz += t * sz;
    }
    if (net) imbalance = net[i];
    const float value = csum_value(c);
    cell[3 * N + i] = i == reference ? 2.0f * value : value;
    cell[7 * N + i] = hx;
    cell[8 * N + i] = hy;
    cell[9 * N + i] = hz;
    r[i] = gx;
    r[N + i] = gy;
    r[2 * N + i] = gz;
    b[i] = make_float4(ru[i], rv[i], rw[i], -continuity_scale * imbalance);
  }
}

// Per face: (sx, sy, sz, Rhie-Chow coefficient), the face half of the fine
// row's continuity term.
__global__ void k_cpl_face_records(int nf, const float* __restrict__ sx,
                                   const float* __restrict__ sy, const float* __restrict__ sz,
                                   const float* __restrict__ coefficient,
                                   float4* __restrict__ face) {
  pdl_entry();
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x)
    face[f] = make_float4(sx[f], sy[f], sz[f], coefficient[f]);
}

// coupled_fine_schur (fv_coupled.kern.h:210-223), cs into plane 19, and
// coupled_fine_coefficients (:229-256), the block inverse and the five
// directed-edge coefficients as the per-cell records and the ELL slots of the
// fine operator, in one pass over each cell's faces (as two kernels 163 us at
// 884,736 hexes, this 125).
__global__ void k_cpl_fine_pack(int n, int width, FineGeometry m, const float* __restrict__ mu,
                                const float* __restrict__ diffusion,
                                const float* __restrict__ mass, const float* __restrict__ weight,
                                const float* __restrict__ r, float* cell, CoupledFine op,
                                float wc) {
  pdl_entry();
  const std::size_t N = n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float q00 = wc * cell[10 * N + i], q01 = wc * cell[11 * N + i], q02 = wc * cell[12 * N + i];
    const float q10 = wc * cell[13 * N + i], q11 = wc * cell[14 * N + i], q12 = wc * cell[15 * N + i];
    const float q20 = wc * cell[16 * N + i], q21 = wc * cell[17 * N + i], q22 = wc * cell[18 * N + i];
    const float half_wc = 0.5f * wc;
    float sum = 0.0f;
    int slot = 0;
    for (int j = m.offsets[i]; j < m.offsets[i + 1] && slot < width; ++j) {
      const int c = m.adjacent[j];
      if (c < 0) continue;
      const int f = m.faces[j];
      const float s = m.sign[j], share = share_of(weight, i, c);
      const float sx = m.sx[f], sy = m.sy[f], sz = m.sz[f];
      sum += wc * share *
             (fabsf(sx) * r[c] / cell[c] + fabsf(sy) * r[N + c] / cell[N + c] +
              fabsf(sz) * r[2 * N + c] / cell[2 * N + c]);
      const float a = -mu[f] * diffusion[f] + fminf(s * mass[f], 0.0f);
      const float bx = half_wc * s * sx, by = half_wc * s * sy, bz = half_wc * s * sz;
      const float gx = bx + q00 * m.dx[j] + q01 * m.dy[j] + q02 * m.dz[j];
      const float gy = by + q10 * m.dx[j] + q11 * m.dy[j] + q12 * m.dz[j];
      const float gz = bz + q20 * m.dx[j] + q21 * m.dy[j] + q22 * m.dz[j];
      const std::size_t k = slot * N + i;
      op.edge[k] = make_float4(a, gx, gy, gz);
      op.edge_h[k] = wc * s * share;
      op.link[k] = make_int2(c, f);
      ++slot;
    }
    for (; slot < width; ++slot) op.link[slot * N + i] = make_int2(-1, 0);
    cell[19 * N + i] = sum;
    const float du = cell[i], dv = cell[N + i], dw = cell[2 * N + i], cd = cell[3 * N + i];
    const float ex = wc * cell[4 * N + i], ey = wc * cell[5 * N + i], ez = wc * cell[6 * N + i];
    const float hx = wc * cell[7 * N + i], hy = wc * cell[8 * N + i], hz = wc * cell[9 * N + i];
    const BlockInverse inv = block_prepare(du, dv, dw, ex, ey, ez, hx, hy, hz, cd + sum);
    op.diag[i] = make_float4(du, dv, dw, cd);
    op.coupling[i] = make_float4(ex, ey, ez, hx);
    op.coupling_yz[i] = make_float2(hy, hz);
    op.schur[i] = inv.schur;
  }
}

// The fine row kernels are bounded to 32 registers (8 resident blocks of 256
// per SM), so the fixed 1,184-block grid runs in one wave: at 40 registers
// the sweep took 142.5 us at 128^3, bounded 122.7 us (0.92 of the measured
// copy bandwidth). The coarse-level and Galerkin kernels are not bounded: the
// spills cost them more than the second wave.
//
// (J x)_i of the fine level (fv_coupled.kern.h:258-278, coupled_fine_row).
__device__ __forceinline__ float4 fine_row(int i, int n, int width, const CoupledFine& op,
                                           const float4* __restrict__ x) {
  const float4 xi = x[i];
  const float4 d = op.diag[i], e = op.coupling[i];
  const float2 h = op.coupling_yz[i];
  float yu = d.x * xi.x + e.x * xi.w;
  float yv = d.y * xi.y + e.y * xi.w;
  float yw = d.z * xi.z + e.z * xi.w;
  float yp = d.w * xi.w + e.w * xi.x + h.x * xi.y + h.y * xi.z;
  const std::size_t N = n;
  for (int s = 0; s < width; ++s) {
    const int2 l = op.link[s * N + i];
    if (l.x < 0) break;
    const float4 g = op.edge[s * N + i];
    const float hs = op.edge_h[s * N + i];
    const float4 sf = op.face[l.y];
    const float4 xc = x[l.x];
    yu += g.x * xc.x + g.y * xc.w;
    yv += g.x * xc.y + g.z * xc.w;
    yw += g.x * xc.z + g.w * xc.w;
    yp += hs * (sf.x * xc.x + sf.y * xc.y + sf.z * xc.z) - sf.w * xc.w;
  }
  return make_float4(yu, yv, yw, yp);
}

__global__ void __launch_bounds__(kBlock, 8) k_cpl_fine_spmv(int n, int width, CoupledFine op,
                                                          const float4* __restrict__ x,
                                                          float4* __restrict__ y) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = fine_row(i, n, width, op, x);
}

// y = J x with the BiCGStab's reduction of y fused in: w.y and alpha, or (kDual)
// y.y, y.w and omega. The FP64 sums need more than 32 registers, so the grid is
// sized for six blocks per SM (still one wave). A cell's four products are added
// before the running sum, a component at a time in the separate reduction, so the
// two may differ in the last bits of FP64.
constexpr int kDotBlocks = 6;
template <bool kDual>
__global__ void __launch_bounds__(kBlock, kDotBlocks)
    k_cpl_fine_spmv_dot(int n, int width, CoupledFine op, const float4* __restrict__ x,
                        const float4* __restrict__ w, float4* __restrict__ y, DeviceReducer red,
                        float* scalars, int* status) {
  pdl_entry();
  if (status[0] != 0) return;
  double a = 0.0, b = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 v = fine_row(i, n, width, op, x), u = w[i];
    y[i] = v;
    const double dot = static_cast<double>(u.x) * v.x + static_cast<double>(u.y) * v.y +
                       static_cast<double>(u.z) * v.z + static_cast<double>(u.w) * v.w;
    if (kDual) {
      a += static_cast<double>(v.x) * v.x + static_cast<double>(v.y) * v.y +
           static_cast<double>(v.z) * v.z + static_cast<double>(v.w) * v.w;
      b += dot;
    } else {
      a += dot;
    }
  }
  finish(as_reducer(red), a, b, kDual, scalars, 2, status,
         kDual ? Epilogue::BicgOmega : Epilogue::BicgAlpha);
}

__global__ void __launch_bounds__(kBlock, 8) k_cpl_fine_residual(int n, int width, CoupledFine op,
                                                              const float4* __restrict__ x,
                                                              const float4* __restrict__ b,
                                                              float4* __restrict__ r) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 y = fine_row(i, n, width, op, x);
    const float4 bi = b[i];
    r[i] = make_float4(bi.x - y.x, bi.y - y.y, bi.z - y.z, bi.w - y.w);
  }
}

// Damped block Jacobi (fv_coupled.kern.h:294-309, coupled_fine_smooth);
// first: x is zero and is not read.
__global__ void __launch_bounds__(kBlock, 8) k_cpl_fine_smooth(int n, int width, CoupledFine op,
                                                            const float4* __restrict__ x,
                                                            const float4* __restrict__ b,
                                                            float4* __restrict__ next, float omega,
                                                            int first) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 r = b[i];
    float4 base = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!first) {
      const float4 y = fine_row(i, n, width, op, x);
      r = make_float4(r.x - y.x, r.y - y.y, r.z - y.z, r.w - y.w);
      base = x[i];
    }
    // The block inverse's factors again from the diagonal (block_prepare's
    // operations): three reciprocals per cell instead of 28 bytes. The records
    // are read again (from L1) rather than held in registers over the row.
    asm volatile("" ::: "memory");
    const float4 m = op.diag[i], e = op.coupling[i];
    const float2 h = op.coupling_yz[i];
    const float iu = 1.0f / m.x, iv = 1.0f / m.y, iw = 1.0f / m.z;
    const float4 d = block_solve(r, e.x, e.y, e.z, iu, iv, iw, e.w * iu, h.x * iv, h.y * iw,
                                 op.schur[i]);
    next[i] = damped(base, d, omega);
  }
}

// fv_coupled.kern.h:554-567: prolongation adds the aggregate's correction.
__global__ void __launch_bounds__(kBlock, 8) k_cpl_prolong(int nf, const int* __restrict__ aggregate,
                              const float4* __restrict__ coarse, float4* __restrict__ fine) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += gridDim.x * blockDim.x) {
    const float4 c = coarse[aggregate[i]];
    float4 v = fine[i];
    v.x += c.x;
    v.y += c.y;
    v.z += c.z;
    v.w += c.w;
    fine[i] = v;
  }
}

// ---- the update of the flow fields --------------------------------------------

// fv_coupled.kern.h:571-578 (coupled_update).
__global__ void k_cpl_update(int n, const float4* __restrict__ delta, float* __restrict__ u,
                             float* __restrict__ v, float* __restrict__ w, float* __restrict__ p,
                             float alpha_u, float alpha_p) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 d = delta[i];
    u[i] += alpha_u * d.x;
    v[i] += alpha_u * d.y;
    w[i] += alpha_u * d.z;
    p[i] += alpha_p * d.w;
  }
}

// Knuth's two-sum and the slack-held pair addition (prelude.h:103-149,
// kpair_add).
struct Pair2 {
  float hi, lo;
};
__device__ __forceinline__ Pair2 two_sum(float a, float b) {
  const float sum = a + b;
  const float part = sum - a;
  return Pair2{sum, (a - (sum - part)) + (b - part)};
}
__device__ __forceinline__ Pair2 pair_add(float hi, float lo, float d, float slack) {
  const float low = lo + d;
  if (fabsf(low) <= slack) return Pair2{hi, low};
  const Pair2 s = two_sum(hi, d);
  return two_sum(s.hi, s.lo + lo);
}

// fv_coupled.kern.h:582-591 (coupled_paired_update).
__global__ void k_cpl_paired_update(int n, const float4* __restrict__ delta, float* __restrict__ u,
                                    float* __restrict__ v, float* __restrict__ w,
                                    float* __restrict__ p, float* __restrict__ u_lo,
                                    float* __restrict__ v_lo, float* __restrict__ w_lo,
                                    float* __restrict__ p_lo, float alpha_u, float alpha_p,
                                    float velocity_slack, float pressure_slack) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 d = delta[i];
    Pair2 x = pair_add(u[i], u_lo[i], alpha_u * d.x, velocity_slack);
    u[i] = x.hi;
    u_lo[i] = x.lo;
    x = pair_add(v[i], v_lo[i], alpha_u * d.y, velocity_slack);
    v[i] = x.hi;
    v_lo[i] = x.lo;
    x = pair_add(w[i], w_lo[i], alpha_u * d.z, velocity_slack);
    w[i] = x.hi;
    w_lo[i] = x.lo;
    x = pair_add(p[i], p_lo[i], alpha_p * d.w, pressure_slack);
    p[i] = x.hi;
    p_lo[i] = x.lo;
  }
}

// The closed-domain gauge (fv_coupled.kern.h:592-620): the reference cell's
// value is picked into `value` by one thread, then subtracted everywhere.
__global__ void k_cpl_pick(const float* __restrict__ p, const float* __restrict__ p_lo,
                           float* __restrict__ value, int index) {
  pdl_entry();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    value[0] = p[index];
    value[1] = p_lo ? p_lo[index] : 0.0f;
  }
}
__global__ void k_cpl_gauge(int n, const float* __restrict__ value, float* __restrict__ p) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    p[i] -= value[0];
}
__global__ void k_cpl_paired_gauge(int n, const float* __restrict__ value, float* __restrict__ p,
                                   float* __restrict__ p_lo, float pressure_slack) {
  pdl_entry();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const Pair2 x = pair_add(p[i], p_lo[i], -(value[0] + value[1]), pressure_slack);
    p[i] = x.hi;
    p_lo[i] = x.lo;
  }
}

FineGeometry geometry(const CoupledMeshDevice& m) {
  return FineGeometry{m.offsets, m.faces, m.sign, m.adjacent, m.sx, m.sy, m.sz, m.dx, m.dy, m.dz};
}

}  // namespace

namespace launch {

void cpl_copy_diagonal(int n, const int* rows, const int* diag, const float* values,
                       const float* physical, float* plane, float inverse_courant, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_cpl_copy_diagonal, grid_for(n), kBlock, 0, s, n, rows, diag, values, physical, plane,
      inverse_courant);
}

void cpl_assemble(const CoupledMeshDevice& m, const CoupledSolveInputs& in, float* cell,
                  float* coefficient, float4* b, float* scratch, CoupledFine op, float wc,
                  float coefficient_scale, float continuity_scale, int reference,
                  cudaStream_t s) {
  const int n = m.n, nf = m.n_faces;
  if (n <= 0) return;
  const FineGeometry g = geometry(m);
  counter += 4;
  pdl(k_cpl_face_coefficient, grid_for(nf), kBlock, 0, s, nf, m.n_internal, m.owner,
      m.neighbour, m.kind, m.diffusion, m.volume, in.physical_diagonal, coefficient,
      coefficient_scale);
  pdl(k_cpl_cell_sums, grid_for(n), kBlock, 0, s, n, m.n_internal, g, m.kind, in.face_weights,
      static_cast<const float*>(coefficient), in.mass, in.net_outflow, in.ru, in.rv, in.rw, cell,
      scratch, b, reference, continuity_scale, wc);
  pdl(k_cpl_face_records, grid_for(nf), kBlock, 0, s, nf, m.sx, m.sy, m.sz,
      static_cast<const float*>(coefficient), const_cast<float4*>(op.face));
  pdl(k_cpl_fine_pack, grid_for(n), kBlock, 0, s, n, m.width, g, in.viscosity, m.diffusion,
      in.mass, in.face_weights, static_cast<const float*>(scratch), cell, op, wc);
}

void cpl_fine_spmv(int n, const CoupledFine& op, int width, const float4* x, float4* y,
                   cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_cpl_fine_spmv, grid_for(n), kBlock, 0, s, n, width, op, x, y);
}

void cpl_fine_spmv_dot(int n, const CoupledFine& op, int width, const float4* x, const float4* w,
                       float4* y, bool dual, DeviceReducer red, float* scalars, int* status,
                       cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  const int grid = std::min(grid_for(n), kSms * kDotBlocks);
  if (dual)
    pdl(k_cpl_fine_spmv_dot<true>, grid, kBlock, 0, s, n, width, op, x, w, y, red, scalars, status);
  else
    pdl(k_cpl_fine_spmv_dot<false>, grid, kBlock, 0, s, n, width, op, x, w, y, red, scalars,
        status);
}

void cpl_fine_residual(int n, const CoupledFine& op, int width, const float4* x, const float4* b,
                       float4* r, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_cpl_fine_residual, grid_for(n), kBlock, 0, s, n, width, op, x, b, r);
}

void cpl_fine_smooth(int n, const CoupledFine& op, int width, const float4* x, const float4* b,
                     float4* next, float omega, bool first, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_cpl_fine_smooth, grid_for(n), kBlock, 0, s, n, width, op, x, b, next, omega,
      first ? 1 : 0);
}

void cpl_prolong(int nf, const int* aggregate, const float4* coarse, float4* fine,
                 cudaStream_t s) {
  if (nf <= 0) return;
  ++counter;
  pdl(k_cpl_prolong, grid_for(nf), kBlock, 0, s, nf, aggregate, coarse, fine);
}

void cpl_update(int n, const float4* delta, float* u, float* v, float* w, float* p, float alpha_u,
                float alpha_p, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_cpl_update, grid_for(n), kBlock, 0, s, n, delta, u, v, w, p, alpha_u, alpha_p);
}

void cpl_paired_update(int n, const float4* delta, float* u, float* v, float* w, float* p,
                       float* u_lo, float* v_lo, float* w_lo, float* p_lo, float alpha_u,
                       float alpha_p, float velocity_slack, float pressure_slack, cudaStream_t s) {
  if (n <= 0) return;
  ++counter;
  pdl(k_cpl_paired_update, grid_for(n), kBlock, 0, s, n, delta, u, v, w, p, u_lo, v_lo, w_lo,
      p_lo, alpha_u, alpha_p, velocity_slack, pressure_slack);
}

void cpl_gauge(int n, float* p, float* p_lo, float pressure_slack, float* value, int index,
               cudaStream_t s) {
  if (n <= 0) return;
  counter += 2;
  pdl(k_cpl_pick, 1, 32, 0, s, static_cast<const float*>(p), static_cast<const float*>(p_lo),
      value, index);
  if (p_lo)
    pdl(k_cpl_paired_gauge, grid_for(n), kBlock, 0, s, n, static_cast<const float*>(value), p,
        p_lo, pressure_slack);
  else
    pdl(k_cpl_gauge, grid_for(n), kBlock, 0, s, n, static_cast<const float*>(value), p);
}

}  // namespace launch
}  // namespace kb2
