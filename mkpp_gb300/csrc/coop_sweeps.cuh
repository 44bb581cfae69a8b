// The differentiation kernels of solver.cuh with a whole warp per cell: the
// checkpointed forward, the discrete adjoint and the tangent.  A block is one
// warp, so that a call of a few cells spreads over all SMs, and a step takes a
// warp a fifth of a lane's time.  Results are bit-identical to the lanes'.
#pragma once
#include "solver.cuh"

namespace mkpp {

// The warp's next cell, ncells or more after the last: from a work counter in
// the workspace, or, where the lanes' form has no use for the workspace, so that
// calls on several streams may share one, the block's own.  (Blocks of one
// cell each cost small_strato's tangent of 6000 and 8000 cells 5%.)
__device__ __forceinline__ size_t sweep_cell(unsigned* next, unsigned lane, unsigned pass, size_t ncells) {
  if (next) return next_cell(next, lane);
  return pass == 0 ? blockIdx.x : ncells;
}

// integrate_checkpoint_kernel.
template <class Mech>
__global__ void __launch_bounds__(32) checkpoint_coop_kernel(LaunchArgs a, CheckpointArgs ck) {
  extern __shared__ double smem[];
  double* S = smem;
  const unsigned lane = threadIdx.x;
  const size_t n = (size_t)a.ncells;
  Mech::coop_constants(S, lane);
  for (unsigned pass = 0; pass <= (unsigned)a.ncells; ++pass) {
    const size_t c = sweep_cell(a.coop_next, lane, pass, n);
    if (c >= n) break;
    if (a.status && a.status[c] != CELL_SUCCESS) {
      if (lane == 0) {
        ck.n[c] = 0;  // no accepted step to revisit
        clear_counts(a, c);
      }
      continue;
    }
    for (int i = lane; i < Mech::NV; i += 32) S[Mech::Y + i] = a.conc[c + n * Mech::var_phys(i)];
    for (int r = lane; r < Mech::NR; r += 32) S[Mech::KT + r] = a.ktab[c + n * r];
    __syncwarp();
    Controller ctl;
    ctl.start(a.dt, a.seed);
    int nacc = 0, nrej = 0, cnt = 0;
    bool capped = false, zero_pivot = false, overflow = false;
    while (ctl.running()) {
      if (ctl.attempts >= a.max_attempts) {
        capped = true;
        break;
      }
      const double h = ctl.next_h();
      int st = 0;
      const double err = Mech::attempt_coop(S, h, st, lane, WarpProgram<Mech::PIVOT_EVERY>());
      zero_pivot |= st != 0;
      if (ctl.update<Mech>(err)) {
        if (cnt >= ck.cap) {
          overflow = true;
          break;
        }
        for (int i = lane; i < Mech::NV; i += 32) {
          ck.y[((size_t)cnt * Mech::NV + i) * n + c] = S[Mech::Y + i];
          S[Mech::Y + i] += S[Mech::DY + i];
        }
        __syncwarp();
        if (lane == 0) ck.h[(size_t)cnt * n + c] = h;
        ++cnt;
        ++nacc;
      } else {
        ++nrej;
      }
    }
    bool fin = true;
    for (int i = lane; i < Mech::NV; i += 32) {
      fin = fin && finite(S[Mech::Y + i]);
      a.conc[c + n * Mech::var_phys(i)] = S[Mech::Y + i];
    }
    fin = __all_sync(0xffffffffu, fin);
    if (lane == 0) {
      ck.n[c] = cnt;
      if (a.status)
        a.status[c] = overflow ? CELL_ERR_CHECKPOINT_OVERFLOW : coop_status(fin, capped, zero_pivot);
      if (a.n_accept) a.n_accept[c] = nacc;
      if (a.n_reject) a.n_reject[c] = nrej;
    }
    __syncwarp();
  }
}

// adjoint_kernel: the step's stages again, then the warp's adjoint program.
template <class Mech>
__global__ void __launch_bounds__(32) adjoint_coop_kernel(AdjointArgs a, CheckpointArgs ck, unsigned* next) {
  extern __shared__ double smem[];
  double* S = smem;
  const unsigned lane = threadIdx.x;
  const size_t n = (size_t)a.ncells;
  Mech::coop_constants(S, lane);
  Mech::adjoint_constants(S, lane);
  for (unsigned pass = 0; pass <= (unsigned)a.ncells; ++pass) {
    const size_t c = sweep_cell(next, lane, pass, n);
    if (c >= n) break;
    for (int r = lane; r < Mech::NR; r += 32) {
      S[Mech::KT + r] = __ldg(a.ktab + (size_t)r * n + c);
      S[Mech::W_KB + r] = 0.0;
    }
    for (int i = lane; i < Mech::NV; i += 32) S[Mech::W_LAM + i] = a.lam[c + n * Mech::var_phys(i)];
    for (int s = ck.count(c) - 1; s >= 0; --s) {
      for (int i = lane; i < Mech::NV; i += 32) S[Mech::Y + i] = ck.y[((size_t)s * Mech::NV + i) * n + c];
      __syncwarp();
      int st = 0;
      Mech::stages_coop(S, ck.h[(size_t)s * n + c], st, lane, WarpProgram<Mech::PIVOT_EVERY>());
      Mech::adjoint_coop(S, lane, WarpProgram<Mech::PIVOT_EVERY>());
    }
    for (int i = lane; i < Mech::NS; i += 32) a.grad_conc[c + n * i] = 0.0;
    __syncwarp();
    for (int i = lane; i < Mech::NV; i += 32) a.grad_conc[c + n * Mech::var_phys(i)] = S[Mech::W_LAM + i];
    for (int r = lane; r < Mech::NR; r += 32) a.grad_k[c + n * r] = S[Mech::W_KB + r];
    __syncwarp();
  }
}

// tangent_kernel: the step's stages again, then the warp's tangent program.
template <class Mech>
__global__ void __launch_bounds__(32) tangent_coop_kernel(TangentArgs a, CheckpointArgs ck, unsigned* next) {
  extern __shared__ double smem[];
  double* S = smem;
  const unsigned lane = threadIdx.x;
  const size_t n = (size_t)a.ncells;
  Mech::coop_constants(S, lane);
  Mech::tangent_constants(S, lane);
  for (unsigned pass = 0; pass <= (unsigned)a.ncells; ++pass) {
    const size_t c = sweep_cell(next, lane, pass, n);
    if (c >= n) break;
    for (int r = lane; r < Mech::NR; r += 32) {
      S[Mech::KT + r] = __ldg(a.ktab + (size_t)r * n + c);
      S[Mech::W_DKR + r] = a.dk ? __ldg(a.dk + (size_t)r * n + c) : 0.0;
    }
    for (int i = lane; i < Mech::NV; i += 32) S[Mech::W_DYT + i] = a.dconc0[c + n * Mech::var_phys(i)];
    const int cnt = ck.count(c);
    for (int s = 0; s < cnt; ++s) {
      for (int i = lane; i < Mech::NV; i += 32) S[Mech::Y + i] = ck.y[((size_t)s * Mech::NV + i) * n + c];
      __syncwarp();
      int st = 0;
      Mech::stages_coop(S, ck.h[(size_t)s * n + c], st, lane, WarpProgram<Mech::PIVOT_EVERY>());
      Mech::tangent_coop(S, lane, WarpProgram<Mech::PIVOT_EVERY>());
    }
    for (int i = lane; i < Mech::NS; i += 32) a.dconc[c + n * i] = 0.0;
    __syncwarp();
    for (int i = lane; i < Mech::NV; i += 32) a.dconc[c + n * Mech::var_phys(i)] = S[Mech::W_DYT + i];
    __syncwarp();
  }
}

}  // namespace mkpp
