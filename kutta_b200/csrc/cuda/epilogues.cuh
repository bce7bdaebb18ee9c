// Grid-wide FP64 reductions that end in one of the reference's single-thread
// scalar updates (compiled with --fmad=false).
#pragma once

#include "common.cuh"
#include "kernels.hpp"

namespace kb2::dev {

__device__ __forceinline__ Reducer as_reducer(DeviceReducer r) {
  return Reducer{r.partials, r.ticket};
}

// ---- scalar updates, src/kutta/kernels/scalars.kern.h:51-121 -----------------
__device__ __forceinline__ void epilogue(Epilogue e, float* sc, int* st) {
  switch (e) {
    case Epilogue::None:
      return;
    case Epilogue::PcgAlpha: {  // solver_pcg_alpha :63-71
      if (st[0] != 0) return;
      const Pair rho = kp_load(sc, 0), pq = kp_load(sc, 2);
      const Pair alpha = kp_div(rho, pq);
      if (!kp_positive(rho) || !kp_positive(pq) || !kp_coefficient(alpha) || kp_zero(alpha))
        st[0] = 2;
      else
        kp_store(sc, 8, alpha);
      return;
    }
    case Epilogue::PcgBeta:
    case Epilogue::PcgBetaFlexible: {  // solver_pcg_beta :72-80
      if (st[0] != 0) return;
      const Pair next = kp_load(sc, 4);
      const Pair numer = e == Epilogue::PcgBetaFlexible
                             ? kp_neg(kp_mul(kp_load(sc, 8), kp_load(sc, 6)))
                             : next;
      const Pair beta = kp_div(numer, kp_load(sc, 0));
      if (!kp_positive(next) || !kp_coefficient(beta) || (kp_zero(beta) && !kp_zero(numer)))
        st[0] = 2;
      else {
        kp_store(sc, 10, beta);
        kp_store(sc, 0, next);
      }
      return;
    }
    case Epilogue::BicgBeta: {  // solver_bicg_beta :81-89
      if (st[0] != 0) return;
      const Pair rho = kp_load(sc, 0), omega = kp_load(sc, 12);
      const Pair beta = kp_mul(kp_div(rho, kp_load(sc, 14)), kp_div(kp_load(sc, 8), omega));
      if (kp_zero(rho) || !kp_finite(rho) || kp_zero(omega) || !kp_coefficient(omega) ||
          !kp_coefficient(beta) || kp_zero(beta))
        st[0] = 2;
      else {
        kp_store(sc, 10, beta);
        st[2] = 0;
      }
      return;
    }
    case Epilogue::BicgAlpha: {  // solver_bicg_alpha :90-97
      if (st[0] != 0) return;
      const Pair rv = kp_load(sc, 2);
      const Pair alpha = kp_div(kp_load(sc, 0), rv);
      if (kp_zero(rv) || !kp_finite(rv) || !kp_coefficient(alpha) || kp_zero(alpha))
        st[0] = 2;
      else
        kp_store(sc, 8, alpha);
      return;
    }
    case Epilogue::BicgS: {  // solver_bicg_s :98-103
      if (st[0] != 0) return;
      ++st[1];
      st[2] = kp_le(kp_load(sc, 16), kp_load(sc, 20)) ? 1 : 0;
      return;
    }
    case Epilogue::BicgOmega: {  // solver_bicg_omega :104-112
      if (st[0] != 0) return;
      if (st[2] != 0) {
        kp_store(sc, 12, kp(0.0f, 0.0f));
        return;
      }
      const Pair tt = kp_load(sc, 2), ts = kp_load(sc, 4);
      const Pair omega = kp_div(ts, tt);
      if (!kp_positive(tt) || !kp_finite(tt) || kp_zero(omega) || !kp_coefficient(omega))
        st[0] = 2;
      else
        kp_store(sc, 12, omega);
      return;
    }
    case Epilogue::CheckPcg:
    case Epilogue::CheckBicg: {  // solver_check :113-121
      if (st[0] != 0) return;
      const bool pcg = e == Epilogue::CheckPcg;
      if (pcg) ++st[1];
      const Pair rr = kp_load(sc, 18);
      if (!kp_finite(rr) || kp_le(rr, kp_load(sc, 20)) || !kp_le(rr, kp_load(sc, 22)) ||
          st[1] % 50 == 0)
        st[0] = 1;
      if (!pcg) kp_store(sc, 14, kp_load(sc, 0));
      return;
    }
  }
}

// Block partial -> grid total -> pair store -> epilogue, in the last block.
__device__ __forceinline__ void finish(const Reducer& red, double a, double b, bool dual,
                                       float* scalars, int offset, int* status, Epilogue epi) {
  __shared__ double shared[32];
  a = block_sum(a, shared);
  if (dual) b = block_sum(b, shared);
  if (!publish(red, a, b, dual)) return;
  const double total_a = gather(red, 0, shared);
  const double total_b = dual ? gather(red, 1, shared) : 0.0;
  if (threadIdx.x == 0) {
    store_pair(scalars, offset, total_a);
    if (dual) store_pair(scalars, offset + 2, total_b);
    epilogue(epi, scalars, status);
    *red.ticket = 0;
  }
}

// The maximum over the grid into check[slot] (NaN wins).
__device__ __forceinline__ void finish_max(const Reducer& red, double worst, double* check,
                                           int slot) {
  __shared__ double shared[32];
  worst = block_max(worst, shared);
  if (!publish(red, worst, 0, false)) return;
  const double total = gather_max(red, shared);
  if (threadIdx.x == 0) {
    check[slot] = total;
    *red.ticket = 0;
  }
}

// BiCGStab's r.r and, for the next update, rhat.r: solver_check, then
// solver_bicg_beta unless the check stopped the iteration (solver.cpp:314-361
// runs the second at the start of the next update, on the same r).
__device__ __forceinline__ void finish_bicg(const Reducer& red, double rr, double rho,
                                            float* scalars, int* status) {
  __shared__ double shared[32];
  rr = block_sum(rr, shared);
  rho = block_sum(rho, shared);
  if (!publish(red, rr, rho, true)) return;
  const double total_rr = gather(red, 0, shared);
  const double total_rho = gather(red, 1, shared);
  if (threadIdx.x == 0) {
    store_pair(scalars, 18, total_rr);
    epilogue(Epilogue::CheckBicg, scalars, status);
    if (status[0] == 0) {
      store_pair(scalars, 0, total_rho);
      epilogue(Epilogue::BicgBeta, scalars, status);
    }
    *red.ticket = 0;
  }
}

}  // namespace kb2::dev
