// Host launchers for the Coupled (4x4-block) solve kernels
// (src/kutta/kernels/fv_coupled.kern.h). Device pointers and sizes only;
// every launcher enqueues on `s` and never synchronises.
#pragma once

#include <cuda_runtime.h>

#include "kernels.hpp"

namespace kb2 {

// The mesh, stencil and least-squares arrays the kernels read, on the device.
struct CoupledMeshDevice {
  int n = 0, n_faces = 0, n_internal = 0;
  int width = 0;  // most internal faces of one cell (ELL slots of the fine operator)
  const int* owner = nullptr;
  const int* neighbour = nullptr;
  const int* offsets = nullptr;   // cell -> its cell-face entries (n + 1)
  const int* faces = nullptr;     // per entry
  const float* sign = nullptr;    // per entry, +1 owner / -1 neighbour
  const int* adjacent = nullptr;  // per entry: the other cell, or -(boundary face + 1)
  const int* kind = nullptr;      // per boundary face
  const float *sx = nullptr, *sy = nullptr, *sz = nullptr;  // face area vectors
  const float *dx = nullptr, *dy = nullptr, *dz = nullptr;  // least-squares rows per entry
  const float* diffusion = nullptr;  // per face
  const float* volume = nullptr;     // per cell
};

// The per-solve flow inputs (device pointers; net_outflow may be null).
struct CoupledSolveInputs {
  const float *ru = nullptr, *rv = nullptr, *rw = nullptr;
  const float* mass = nullptr;
  const float* viscosity = nullptr;
  const float* physical_diagonal = nullptr;
  const float* face_weights = nullptr;
  const float* net_outflow = nullptr;
};

// The fine operator's per-cell records and ELL slots (slot-major: slot s of
// cell i at s n + i); see coupled_kernels.cu.
struct CoupledFine {
  float4* diag;         // (du, dv, dw, cd)
  float4* coupling;     // (wc Gx, wc Gy, wc Gz, wc Hx)
  float2* coupling_yz;  // (wc Hy, wc Hz)
  float* schur;         // the block inverse's Schur denominator
  float4* edge;         // per slot: (a, gx, gy, gz)
  float* edge_h;        // per slot: h
  int2* link;           // per slot: (neighbour, face), neighbour -1 past the row's end
  const float4* face;   // per face: (sx, sy, sz, Rhie-Chow coefficient)
};

// One coarse level: CSR with two float4 per entry, (a, gx, gy, gz) and
// (c, hx, hy, hz) (a of a diagonal entry is 0: its momentum part is in d), and
// 11 planes of n per row (du dv dw cs iu iv iw hx iu hy iv hz iw schur).
struct CoupledLevel {
  int n = 0, nnz = 0;
  const int* rows = nullptr;
  const int* cols = nullptr;
  const int* diag = nullptr;
  float4* entry = nullptr;
  float* d = nullptr;
  // The contributions of each entry's Galerkin sum, in the reference's order:
  // terms [term_at[e], term_at[e + 1]). From the fine level a term is an ELL slot
  // of the fine operator, from a coarse one 2 * entry, + 1 for a diagonal entry;
  // ~row says that a member row's own data comes next (diagonal entries only,
  // whose lists begin with one).
  const int* term_at = nullptr;
  // Where the numbers of terms pass 31 bits, long_terms holds them instead.
  const int* terms = nullptr;
  const long long* long_terms = nullptr;
  const int* term_faces = nullptr;  // from the fine level: each term's face
};

// Level k -> k+1: aggregate of each fine row, member lists of each coarse row.
struct CoupledTransfer {
  const int* aggregate = nullptr;
  const int* offsets = nullptr;
  const int* members = nullptr;
};

// The V-cycle of the small coarse levels, each of at most kMaxRows rows and
// kMaxEntries entries, as one single-block launch: levels 0 .. levels-1 of the
// tail, the first one's right-hand side from b, its correction into x.
struct CoupledTail {
  static constexpr int kMaxLevels = 8;
  static constexpr int kMaxRows = 128, kMaxEntries = 2048;
  int levels = 0;
  int pre = 1, post = 2, coarsest = 8;
  float omega = 0.7f;
  CoupledLevel op[kMaxLevels];
  CoupledTransfer down[kMaxLevels];  // down[k]: tail level k -> k + 1
  const float4* b = nullptr;
  float4* x = nullptr;
};

namespace launch {

// Plane = the cell data's slot k (momentum diagonal of component k).
void cpl_copy_diagonal(int n, const int* rows, const int* diag, const float* values,
                       const float* physical, float* plane, float inverse_courant, cudaStream_t s);
// Face coefficients, H_ii, pressure diagonal and right-hand side b (float4
// per cell), the smoother's Schur bound, the face records and the packed fine
// operator. scratch: 3n floats.
void cpl_assemble(const CoupledMeshDevice& m, const CoupledSolveInputs& in, float* cell,
                  float* coefficient, float4* b, float* scratch, CoupledFine op, float wc,
                  float coefficient_scale, float continuity_scale, int reference, cudaStream_t s);
// Galerkin operators: the fine level's contributions come from its packed
// records (cpl_assemble first), a coarse level's from its entries.
void cpl_galerkin_fine(const CoupledLevel& l, const CoupledFine& op, const float* cell, int cells,
                       float wc, cudaStream_t s);
void cpl_galerkin_coarse(const CoupledLevel& l, const CoupledLevel& f, cudaStream_t s);
// The term lists, a thread per coarse row: first each entry's count of terms,
// then (after an exclusive scan into term_at) the terms. Fine level: its
// adjacency through the mesh; coarse: the level above's CSR. Term is int or long long.
template <class Term>
void cpl_terms_fine(const CoupledLevel& l, const CoupledTransfer& t, const CoupledMeshDevice& m,
                    int* count, Term* terms, int* term_faces, cudaStream_t s);
template <class Term>
void cpl_terms_coarse(const CoupledLevel& l, const CoupledTransfer& t, const CoupledLevel& f,
                      int* count, Term* terms, cudaStream_t s);
// |G| row sums into scratch (3n), then cs and the block inverse.
void cpl_coarse_prepare(const CoupledLevel& l, float* scratch, cudaStream_t s);

void cpl_fine_spmv(int n, const CoupledFine& op, int width, const float4* x, float4* y,
                   cudaStream_t s);
// y = J x, then w.y -> scalars[2] and solver_bicg_alpha, or (dual) y.y, y.w ->
// scalars[2], scalars[4] and solver_bicg_omega; skipped while status[0] != 0.
void cpl_fine_spmv_dot(int n, const CoupledFine& op, int width, const float4* x, const float4* w,
                       float4* y, bool dual, DeviceReducer red, float* scalars, int* status,
                       cudaStream_t s);
void cpl_fine_residual(int n, const CoupledFine& op, int width, const float4* x, const float4* b,
                       float4* r, cudaStream_t s);
void cpl_fine_smooth(int n, const CoupledFine& op, int width, const float4* x, const float4* b,
                     float4* next, float omega, bool first, cudaStream_t s);
void cpl_coarse_residual(const CoupledLevel& l, const float4* x, const float4* b, float4* r,
                         cudaStream_t s);
// One sweep; with aggregate != null from x + coarse[aggregate] (the prolongation
// folded in).
void cpl_coarse_smooth(const CoupledLevel& l, const float4* x, const float4* b, float4* next,
                       float omega, bool first, const int* aggregate, const float4* coarse,
                       cudaStream_t s);
// coarse = the sum of each aggregate's members; with next != null also level
// l's (the coarse one's) first sweep from zero.
void cpl_restrict(int nc, const int* offsets, const int* members, const float4* fine,
                  float4* coarse, const CoupledLevel* l, float omega, float4* next,
                  cudaStream_t s);
void cpl_prolong(int nf, const int* aggregate, const float4* coarse, float4* fine,
                 cudaStream_t s);

void cpl_tail(const CoupledTail& t, cudaStream_t s);

void cpl_update(int n, const float4* delta, float* u, float* v, float* w, float* p, float alpha_u,
                float alpha_p, cudaStream_t s);
void cpl_paired_update(int n, const float4* delta, float* u, float* v, float* w, float* p,
                       float* u_lo, float* v_lo, float* w_lo, float* p_lo, float alpha_u,
                       float alpha_p, float velocity_slack, float pressure_slack, cudaStream_t s);
// p -= p[index] (or, with p_lo, the pair's value at index, slack-held);
// value: 2 floats of device scratch.
void cpl_gauge(int n, float* p, float* p_lo, float pressure_slack, float* value, int index,
               cudaStream_t s);

}  // namespace launch
}  // namespace kb2
