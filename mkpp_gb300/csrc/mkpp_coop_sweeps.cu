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

// Up to as many cells as a plain integrate; register stores longer: small_strato's
// gradient 6.3 against 6.6 ms for 2000 cells, 11.3 against 9.7 for 4325, and its
// tangent, whose lanes walk a program on the global tile, 9.6 ms for 4325 cells
// and 13.5 for 8000 against 14 on lanes.
bool sweep_on_warps(size_t cells, bool tangent) {
  constexpr size_t kRegister = Mech::NLU > 20 ? 2000 : 300, kTangent = Mech::NLU > 20 ? 8000 : 300;
  const size_t most = coop_cells() == 0 ? 0
                      : StoreInfo::kTile ? (size_t)coop_cells()
                                         : (tangent ? kTangent : kRegister);
  return kSlots * sizeof(double) <= kMaxSmem && cells <= most;
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
