// The differentiation kernels with a warp per cell, of one mechanism library.
#include "capi_common.cuh"
#include "coop_sweeps.cuh"

namespace mkpp_tu {

namespace {

// Launches `kernel` with one warp per block: with a work counter, as many as
// the cells and the shared memory of the SMs allow, else a block per cell.
template <class Kernel, class... Args>
int launch_warps(Kernel kernel, size_t slots, int cells, unsigned* next, cudaStream_t stream, const Args&... args) {
  const size_t smem = slots * sizeof(double);
  if (!allow_smem(kernel, smem)) return MKPP_ERROR_DEVICE;
  int blocks = cells;
  if (next) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32, smem) != cudaSuccess || per_sm < 1)
      return MKPP_ERROR_DEVICE;
    if (cudaMemsetAsync(next, 0, sizeof(unsigned), stream) != cudaSuccess) return MKPP_ERROR_DEVICE;
    blocks = std::min(cells, per_sm * sm_count());
  }
  kernel<<<blocks, 32, smem, stream>>>(args...);
  return cudaGetLastError() == cudaSuccess ? MKPP_SUCCESS : MKPP_ERROR_DEVICE;
}

constexpr size_t kSlots = std::max(std::max(Mech::WARP_SLOTS, Mech::ADJ_COOP_SLOTS), Mech::TLM_COOP_SLOTS);

}  // namespace

// Up to this many cells; the lanes' time hardly depends on their number until
// they fill the SMs.  Warps against lanes:
//   SAPRC99's gradient: 2048 cells 88 against 484 ms, 10000 cells 165 against 485;
//   saprc99_mini's: 4000 cells 4.3 against 10.7 ms, 8000 cells 5.2 against 10.3;
//   register stores: small_strato's gradient 6.3 against 9.5 ms for 2000 cells,
//   11.3 against 9.7 for 4325, its tangent, whose lanes walk a program on the
//   global tile, 9.3 against 14.5 ms for 4000 cells and 13.6 against 14.5 for
//   8000; Chapman's gradient 1.35 against 1.57 ms for 300 cells;
//   TS1, whose lanes walk programs everywhere, nine steps a cell: the forward
//   134 against 284 ms for 16384 cells, 494 against 639 for 65536; the adjoint,
//   whose store leaves room for two warps per SM, 271 against 339 ms for 12000
//   cells, 366 against 370 for 16384, 895 against 606 for 40000; the tangent,
//   three warps per SM, 250 against 368 ms for 16384, 401 against 403 for 26000,
//   610 against 601 for 40000, 998 against 843 for 65536.
bool sweep_on_warps(size_t cells, Sweep sweep) {
  constexpr bool kLargeRegister = Mech::NLU > 20;
  size_t most;
  if (Mech::TABLE_ATTEMPT)
    most = sweep == Sweep::kForward ? SIZE_MAX : sweep == Sweep::kAdjoint ? 16384 : 26000;
  else if (StoreInfo::kTile)
    most = Mech::LU_FMA > 2000 ? 14000 : 10000;
  else
    most = !kLargeRegister ? 300 : sweep == Sweep::kTangent ? 8000 : 2000;
  return coop_cells() > 0 && kSlots * sizeof(double) <= kMaxSmem && cells <= most;
}

int launch_checkpoint_coop(mkpp::LaunchArgs a, const mkpp::CheckpointArgs& ck, unsigned* next, cudaStream_t stream) {
  if (!mkpp::StoreN<Mech::NSLOTS>::kTile) next = nullptr;
  a.coop_next = next;
  return launch_warps(mkpp::checkpoint_coop_kernel<Mech>, Mech::WARP_SLOTS, a.ncells, next, stream, a, ck);
}

int launch_adjoint_coop(const mkpp::AdjointArgs& a, const mkpp::CheckpointArgs& ck, unsigned* next,
                        cudaStream_t stream) {
  if (!mkpp::StoreN<Mech::NSLOTS_ADJ>::kTile) next = nullptr;
  return launch_warps(mkpp::adjoint_coop_kernel<Mech>, Mech::ADJ_COOP_SLOTS, a.ncells, next, stream, a, ck, next);
}

int launch_tangent_coop(const mkpp::TangentArgs& a, const mkpp::CheckpointArgs& ck, unsigned* next,
                        cudaStream_t stream) {
  return launch_warps(mkpp::tangent_coop_kernel<Mech>, Mech::TLM_COOP_SLOTS, a.ncells, next, stream, a, ck, next);
}

}  // namespace mkpp_tu
