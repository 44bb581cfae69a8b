// Tendency and dense-Jacobian evaluation of one mechanism library
// (compute_rates / compute_jacobian of the reference,
// src/mkpp/templates/kernel_functions/compute_{rates,jacobian}.j2), walking
// the mechanism's evaluation tables (namespace eval of its generated header)
// with the arithmetic of fun() and jac_w().
//
// Both are bound by memory: the Jacobian is NS^2 values per cell written once.
// A block takes 32 cells, one per lane (64 for the Jacobian), and its warps
// share their rates (or one column's partial derivatives) in shared memory and
// divide the rows, so that every output row is one coalesced store per warp and
// a small call still has blocks for all SMs.  A thread per cell, which zero-filled the
// matrix, wrote W and flipped its sign through tables of slot positions on the
// stack, took 92.8 ms for SAPRC99's 20000 cells (1.08 GB); this takes 0.23 ms.
// TS1, 1001 cells: 4.5 -> 0.11 ms, the tendencies 3.1 -> 0.06 ms.
//
// Rates (or partials of a column) that 32 cells have too many of for a block's
// shared memory, above 908, are multiplied out again for each term.
#include "capi_common.cuh"

using namespace mkpp_tu;

namespace {

namespace T = MKPP_MECH_NS::eval;

constexpr int kWarps = 8;       // of a block, one column of the Jacobian
constexpr int kRateWarps = 16;  // of a block, all rates and tendencies
constexpr size_t kRatesSmem = (size_t)T::RATES * 32 * sizeof(double);
constexpr bool kStageRates = kRatesSmem <= kMaxSmem;
constexpr size_t kDefaultSmem = 48 * 1024;

// State accessor over a cell's row of the (species x cells) array.
struct CellState {
  const double* conc;
  size_t c, n;
  __device__ __forceinline__ double operator()(int i) const { return conc[c + n * Mech::var_phys(i)]; }
};

// A mechanism whose store fits in registers: a thread per cell, every output
// written once (small_strato, 262144 cells: the tendencies in 28 us, 36 with
// the tables).
__global__ void __launch_bounds__(128, 1) eval_cell_rates_kernel(size_t n, const double* conc, const double* ktab,
                                                              double* out) {
  const size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  const mkpp::KTable k{ktab + c, n};
  for (int s = 0; s < Mech::NS; ++s) out[c + n * s] = 0.0;
  Mech::fun(CellState{conc, c, n}, k, [&](int i, double v) { out[c + n * Mech::var_phys(i)] = v; });
}

template <class M>
__global__ void __launch_bounds__(128, 1) eval_cell_jacobian_kernel(size_t n, const double* conc, const double* ktab,
                                                                 double* out) {
  const size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  const mkpp::KTable k{ktab + c, n};
  mkpp::RegStore<M::NLU> W;
  M::jac_w(CellState{conc, c, n}, k, 0.0, W);  // -J on the W slots
#pragma unroll
  for (int e = 0; e < M::NS * M::NS; ++e) {
    const int slot = M::w_slot(e);
    out[c + n * e] = slot < 0 ? 0.0 : -W[slot < 0 ? 0 : slot];
  }
}

// k times the coded factors, left to right: species (their concentrations in
// cell c), or POWER + a number.
__device__ __forceinline__ double product(double k, unsigned code, const double* __restrict__ conc, size_t c,
                                          size_t n) {
  const auto* __restrict__ f = T::factor<> + (code >> T::LEN_BITS);
  double v = k;
  for (unsigned i = 0; i < (code & ((1u << T::LEN_BITS) - 1u)); ++i) {
    const unsigned x = __ldg(f + i);
    v *= (x & T::POWER) ? (double)(x & (T::POWER - 1u)) : __ldg(conc + c + n * x);
  }
  return v;
}

// c * t; most coefficients are 1 or -1, which cost no FP64 instruction.
__device__ __forceinline__ double first_term(double c, double t) {
  const long long bits = __double_as_longlong(c);
  return (bits << 1) == (__double_as_longlong(1.0) << 1) ? mkpp::flip_sign(t, (unsigned)(bits >> 32) & 0x80000000u)
                                                         : c * t;
}

__global__ void __launch_bounds__(kRateWarps * 32) eval_rates_kernel(size_t n, const double* __restrict__ conc,
                                                                const double* __restrict__ ktab,
                                                                double* __restrict__ out) {
  extern __shared__ double q[];  // [reaction][lane]
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const size_t cell = blockIdx.x * (size_t)32 + lane;
  const size_t c = cell < n ? cell : n - 1;
  auto product_of = [&](int r) { return product(__ldg(ktab + c + n * r), T::rate<>[r], conc, c, n); };
  if constexpr (kStageRates) {
    for (int r = warp; r < T::RATES; r += kRateWarps) q[r * 32 + lane] = product_of(r);
    __syncthreads();
  }
  auto rate = [&](int r) {
    if constexpr (kStageRates)
      return q[r * 32 + lane];
    else
      return product_of(r);
  };
  for (int i = warp; i < Mech::NS; i += kRateWarps) {
    const int begin = T::f_ptr<>[i], end = T::f_ptr<>[i + 1];
    double v = begin < end ? first_term(T::f_coef<>[begin], rate(T::f_term<>[begin])) : 0.0;
    for (int t = begin + 1; t < end; ++t) v = fma(T::f_coef<>[t], rate(T::f_term<>[t]), v);
    if (cell < n) out[cell + n * i] = v;
  }
}

// Column blockIdx.y of the Jacobian of 32 * kCells cells, kCells per lane, its
// partials in shared memory if kStage.
template <int kCells, bool kStage>
__global__ void __launch_bounds__(kWarps * 32) eval_jacobian_kernel(size_t n, const double* __restrict__ conc,
                                                                   const double* __restrict__ ktab,
                                                                   double* __restrict__ out) {
  extern __shared__ double d[];  // [partial of the column][cell]
  constexpr int kRow = 32 * kCells;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const size_t cell = blockIdx.x * (size_t)kRow + lane;
  const int col = blockIdx.y;
  const int first = T::p_ptr<>[col], count = T::p_ptr<>[col + 1] - first;
  auto product_of = [&](int p, int i) {
    const size_t c = cell + 32 * i < n ? cell + 32 * i : n - 1;
    return product(__ldg(ktab + n * T::p_rate<>[first + p] + c), T::p_product<>[first + p], conc, c, n);
  };
  if constexpr (kStage) {
    for (int p = warp; p < count; p += kWarps) {
#pragma unroll
      for (int i = 0; i < kCells; ++i) d[p * kRow + 32 * i + lane] = product_of(p, i);
    }
    __syncthreads();
  }
  auto partial = [&](int p, int i) {
    if constexpr (kStage)
      return d[p * kRow + 32 * i + lane];
    else
      return product_of(p, i);
  };
  double* column = out + n * (size_t)Mech::NS * col + cell;
  const unsigned* entries = T::j_ptr<> + Mech::NS * col;
  for (int row = warp; row < Mech::NS; row += kWarps) {
    const unsigned entry = entries[row];
    double v[kCells];
#pragma unroll
    for (int i = 0; i < kCells; ++i) v[i] = 0.0;
    if (entry & 2u) {  // -W with 1/(gamma h) = 0, which the diagonal's sum starts from
      const int end = entries[row + 1] >> 2;
      int t = entry >> 2;
      if (!(entry & 1u) && t < end) {
#pragma unroll
        for (int i = 0; i < kCells; ++i) v[i] = first_term(T::j_coef<>[t], partial(T::j_term<>[t], i));
        ++t;
      }
      for (; t < end; ++t) {
#pragma unroll
        for (int i = 0; i < kCells; ++i) v[i] = fma(T::j_coef<>[t], partial(T::j_term<>[t], i), v[i]);
      }
#pragma unroll
      for (int i = 0; i < kCells; ++i) v[i] = -v[i];
    }
#pragma unroll
    for (int i = 0; i < kCells; ++i)
      if (cell + 32 * i < n) column[n * row + 32 * i] = v[i];
  }
}

template <int kCells>
int launch_jacobian(size_t n, const double* conc, const double* ktab, double* out, cudaStream_t stream) {
  constexpr size_t kPartials = (size_t)T::MAX_PARTIALS * 32 * kCells * sizeof(double);
  constexpr bool kStage = kPartials <= kMaxSmem;
  constexpr size_t kSmem = kStage ? kPartials : 0;
  const auto kernel = eval_jacobian_kernel<kCells, kStage>;
  if (kSmem > kDefaultSmem && !allow_smem(kernel, kSmem)) return MKPP_ERROR_DEVICE;
  kernel<<<dim3(launch_grid(n, 32 * kCells), Mech::NS), kWarps * 32, kSmem, stream>>>(n, conc, ktab, out);
  return cudaGetLastError() == cudaSuccess ? MKPP_SUCCESS : MKPP_ERROR_DEVICE;
}

// Columns of the dense Jacobian that belong to fixed species (through the
// rate constants' dependence on them), written straight to the output.
__global__ void __launch_bounds__(128, 1) mkpp_fixed_columns_kernel(size_t n, const double* conc, const double* temp,
                                                                 const double* rho, const double* rh,
                                                                 const double* clw, const double* param,
                                                                 double* out) {
  const size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  const CellState y{conc, c, n};
  const double T = (Mech::RUNTIME_ENV && temp) ? temp[c] : Mech::ENV_T;
  const double RHO = (Mech::RUNTIME_ENV && rho) ? rho[c] : Mech::ENV_RHO;
  const double RH = rh ? rh[c] : 0.5;
  const double CLW = clw ? clw[c] : 0.0;
  const mkpp::CellRow fix{conc + c, n};
  const size_t NS = Mech::NS;
  auto put = [&](int row, int col, double v) { out[c + n * (row + NS * col)] = v; };
  if (param) {
    const mkpp::CellRow P{param + c, n};
    Mech::jac_fixed_columns(P, fix, T, RHO, RH, CLW, y, put);
  } else {
    const mkpp::ZeroRow P;
    Mech::jac_fixed_columns(P, fix, T, RHO, RH, CLW, y, put);
  }
}

}  // namespace

namespace mkpp_tu {

int launch_eval_rates(size_t n, const double* conc, const double* ktab, double* out, cudaStream_t stream) {
  if constexpr (!StoreInfo::kTile) {
    eval_cell_rates_kernel<<<launch_grid(n, 128), 128, 0, stream>>>(n, conc, ktab, out);
    return cudaGetLastError() == cudaSuccess ? MKPP_SUCCESS : MKPP_ERROR_DEVICE;
  }
  constexpr size_t kSmem = kStageRates ? kRatesSmem : 0;
  if (kSmem > kDefaultSmem && !allow_smem(eval_rates_kernel, kSmem)) return MKPP_ERROR_DEVICE;
  eval_rates_kernel<<<launch_grid(n, 32), kRateWarps * 32, kSmem, stream>>>(n, conc, ktab, out);
  return cudaGetLastError() == cudaSuccess ? MKPP_SUCCESS : MKPP_ERROR_DEVICE;
}

int launch_eval_jacobian(size_t n, const double* conc, const double* ktab, double* out, cudaStream_t stream) {
  if constexpr (!StoreInfo::kTile) {
    eval_cell_jacobian_kernel<Mech><<<launch_grid(n, 128), 128, 0, stream>>>(n, conc, ktab, out);
    return cudaGetLastError() == cudaSuccess ? MKPP_SUCCESS : MKPP_ERROR_DEVICE;
  }
  // Two cells per lane halve the table reads of an output (SAPRC99, 20000
  // cells: 279 -> 234 us), but need twice the shared memory (TS1, 30 KB for a
  // column of one cell a lane: 107 -> 137 us for 1001 cells) and enough blocks
  // (100 SAPRC99 cells: 17 us, 23 with two).
  if (T::MAX_PARTIALS <= 96 && n >= 2048) return launch_jacobian<2>(n, conc, ktab, out, stream);
  return launch_jacobian<1>(n, conc, ktab, out, stream);
}

int launch_fixed_columns(size_t n, const double* conc, const double* temp, const double* rho, const double* rh,
                         const double* clw, const double* param, double* out, cudaStream_t stream) {
  mkpp_fixed_columns_kernel<<<launch_grid(n, 128), 128, 0, stream>>>(n, conc, temp, rho, rh, clw, param, out);
  return cudaGetLastError() == cudaSuccess ? MKPP_SUCCESS : MKPP_ERROR_DEVICE;
}

}  // namespace mkpp_tu

extern "C" {

int mkpp_gpu_evaluate_rates(size_t num_cells, const double* conc, const double* ktab, double* rates_out,
                            void* stream) {
  if (!conc || !ktab || !rates_out) return MKPP_ERROR_NULL_POINTER;
  if (num_cells == 0) return MKPP_ERROR_INVALID_ARGUMENT;
  return launch_eval_rates(num_cells, conc, ktab, rates_out, (cudaStream_t)stream);
}

int mkpp_gpu_evaluate_jacobian(size_t num_cells, const double* conc, const double* ktab, double* jac_out,
                               void* stream) {
  if (!conc || !ktab || !jac_out) return MKPP_ERROR_NULL_POINTER;
  if (num_cells == 0) return MKPP_ERROR_INVALID_ARGUMENT;
  return launch_eval_jacobian(num_cells, conc, ktab, jac_out, (cudaStream_t)stream);
}

}  // extern "C"
