// Device-side vocabulary shared by every generated mechanism header and the
// solver kernels: per-cell status codes, strided accessors over the
// cell-innermost (LayoutLeft) arrays, and math constants used by the emitted
// rate-constant expressions.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#ifndef M_LN10
#define M_LN10 2.30258509299404568402
#endif

namespace mkpp {

// Per-cell outcome codes; values follow mkpp_host::CellErrorCode
// (src/mkpp_host/include/mkpp_host/dispatcher.hpp:15-21).
enum CellStatus : int {
  CELL_SUCCESS = 0,
  CELL_ERR_SINGULAR_MATRIX = 1,
  CELL_ERR_NON_FINITE_STATE = 2,
  CELL_ERR_CONVERGENCE_FAILURE = 3,
  CELL_ERR_NUMERICAL_FAILURE = 4,
  CELL_ERR_CHECKPOINT_OVERFLOW = 5,   // more accepted steps than checkpoint slots
};

// Read-only strided view of one cell's row in a LayoutLeft (cells x n) array:
// element s of cell c lives at base[c + ncells * s].
struct CellRow {
  const double* __restrict__ base;
  size_t stride;
  __device__ __forceinline__ double operator()(int s) const { return __ldg(base + (size_t)s * stride); }
};

// Writable strided row of the rate-constant table, which notes whether every
// value was finite.
struct CheckedRowOut {
  double* __restrict__ base;
  size_t stride;
  bool ok;
  __device__ __forceinline__ void set(int r, double v) {
    base[(size_t)r * stride] = v;
    ok = ok && isfinite(v);
  }
};

// Rate constants read back from the (reactions x cells) table.
struct KTable {
  const double* __restrict__ base;
  size_t stride;
  __device__ __forceinline__ double operator()(int r) const { return __ldg(base + (size_t)r * stride); }
};

// Rate constants held in a private array (adjoint / small mechanisms).
template <int N>
struct KLocal {
  double v[N];
  __device__ __forceinline__ double operator()(int r) const { return v[r]; }
  __device__ __forceinline__ void set(int r, double x) { v[r] = x; }
};

__device__ __forceinline__ bool finite(double x) { return isfinite(x); }

// ---------------------------------------------------------------------------
// Programs of uniform operations S[out] = fma(+-S[a], S[b], S[c]) or
// S[out] = 1 / S[b], one 64-bit word each, four 16-bit fields of slot * 4 plus
// two flags (emitter/warp_schedule.py):
//   a: 1 negate the product | b, c: 1 the lane's previous result instead |
//   out: 1 store nothing, 2 reciprocal.
// ---------------------------------------------------------------------------
struct ProgramWord {
  unsigned lo, hi;
  __device__ __forceinline__ ProgramWord(unsigned long long w) : lo((unsigned)w), hi((unsigned)(w >> 32)) {}
  __device__ __forceinline__ unsigned negate() const { return lo << 31; }  // the sign bit
  __device__ __forceinline__ bool prev_b() const { return lo & 0x10000u; }
  __device__ __forceinline__ bool prev_c() const { return hi & 1u; }
  __device__ __forceinline__ bool stores() const { return !(hi & 0x10000u); }
  __device__ __forceinline__ bool reciprocal() const { return hi & 0x20000u; }
  __device__ __forceinline__ unsigned a() const { return (lo >> 2) & 0x3fffu; }
  __device__ __forceinline__ unsigned b() const { return lo >> 18; }
  __device__ __forceinline__ unsigned c() const { return (hi >> 2) & 0x3fffu; }
  __device__ __forceinline__ unsigned out() const { return hi >> 18; }
};

__device__ __forceinline__ double flip_sign(double x, unsigned sign) {
  return __longlong_as_double(__double_as_longlong(x) ^ ((long long)sign << 32));
}
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }

// Sequential form: one thread runs `ops` words on its own store.  Returns
// false if a reciprocal met a zero.
template <class SA>
__device__ __forceinline__ bool run_program(SA& S, const unsigned long long* __restrict__ prog, int ops) {
  double prev = 0.0;
  bool ok = true;
  for (int n = 0; n < ops; ++n) {
    const ProgramWord w(__ldg(prog + n));
    const double B = w.prev_b() ? prev : S[w.b()];
    if (w.reciprocal()) {
      ok = ok && !is_zero(B);
      prev = 1.0 / B;
    } else {
      const double C = w.prev_c() ? prev : S[w.c()];
      prev = fma(flip_sign(S[w.a()], w.negate()), B, C);
    }
    if (w.stores()) S[w.out()] = prev;
  }
  return ok;
}

}  // namespace mkpp
