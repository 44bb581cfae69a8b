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

__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }

// ---------------------------------------------------------------------------
// a / b, correctly rounded, in 32-bit integer arithmetic.
//
// The FP64 pipe of GB300 issues a warp instruction per 64 cycles and a
// division takes it six to nine of them, half of a small mechanism's attempt
// (Chapman: 12 divisions); the integer pipes are idle.  Long division in base
// 2^28: with the significands n and d as integers and X an underestimate of
// 2^62 / (d / 2^22) to 2^-30 (the hardware's FP32 reciprocal and one Newton
// step), two quotient digits (n X, then R X of the remainder) give 56 bits that
// are at most 2 short, which the remainder corrects; the rest is rounding to
// nearest even with the remainder as the sticky bit.  Exponents outside the
// normal range, on either side or in the result, take the hardware's division.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double divide(double a, double b) {
#ifdef __CUDA_ARCH__
  typedef unsigned long long u64;
  const u64 ab = (u64)__double_as_longlong(a), bb = (u64)__double_as_longlong(b);
  const int ea = (int)(ab >> 52) & 0x7ff, eb = (int)(bb >> 52) & 0x7ff;
  const int e = ea - eb + 1023;
  constexpr u64 kOne = 1ull << 52;
  const bool zero = is_zero(a);
  if ((unsigned)(eb - 1) >= 2046u || (!zero && ((unsigned)(ea - 1) >= 2046u || (unsigned)(e - 2) >= 2043u)))
    return a / b;
  const u64 n = (ab & (kOne - 1)) | kOne, d = (bb & (kOne - 1)) | kOne;
  const unsigned D = (unsigned)(d >> 22) + 1u;  // at most 2^31
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(D)));
  const unsigned X0 = __float2uint_rz(r * 4.6116838e18f);  // 2^62 (1 - 2^-21): below 2^62 / D
  const u64 short_of = (1ull << 62) - (u64)X0 * D;         // below 2^42
  const unsigned X = X0 + (unsigned)(((u64)X0 * (unsigned)(short_of >> 10)) >> 52);
  const unsigned q1 = (unsigned)(((u64)(unsigned)(n >> 21) * X) >> 36);
  u64 R = (n << 27) - q1 * d;                              // below 2^55
  const unsigned q2 = (unsigned)(((u64)(unsigned)(R >> 23) * X) >> 33);
  R = (R << 28) - q2 * d;                                  // below 3 d
  u64 q = ((u64)q1 << 28) + q2;
  if (R >= 2 * d) {
    R -= 2 * d;
    q += 2;
  }
  if (R >= d) {
    R -= d;
    q += 1;
  }
  q |= R != 0;
  // q is n / d * 2^55: 56 bits where n >= d, else 55.
  const unsigned top = (unsigned)(q >> 55);
  const unsigned drop = 2u + top;
  const u64 m = (q + ((1u << (drop - 1)) - 1u) + ((q >> drop) & 1u)) >> drop;
  const u64 bits = ((u64)(unsigned)(e - 2 + (int)top) << 52) + m;  // m's leading bit adds one to the exponent
  const u64 sign = (ab ^ bb) & (1ull << 63);
  return __longlong_as_double((long long)((zero ? 0ull : bits) | sign));
#else
  return a / b;
#endif
}

// a < b, and the smaller, of numbers that are zero or positive (not NaN), by
// their bit patterns.
__device__ __forceinline__ bool below(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ double least(double a, double b) { return below(b, a) ? b : a; }
// fmax(x, floor) for a positive floor and x zero, positive or NaN.
__device__ __forceinline__ double at_least(double x, double floor) {
  const long long bits = __double_as_longlong(x);
  return bits > (0x7ffll << 52) || bits < __double_as_longlong(floor) ? floor : x;
}

// A number of the rate expressions whose divisions are divide(): nearly every
// rate constant divides by the temperature.
struct Num {
  double v;
  __device__ __forceinline__ Num(double x) : v(x) {}
  __device__ __forceinline__ friend Num operator+(Num a, Num b) { return a.v + b.v; }
  __device__ __forceinline__ friend Num operator-(Num a, Num b) { return a.v - b.v; }
  __device__ __forceinline__ friend Num operator*(Num a, Num b) { return a.v * b.v; }
  __device__ __forceinline__ friend Num operator/(Num a, Num b) { return divide(a.v, b.v); }
  __device__ __forceinline__ friend Num operator-(Num a) { return -a.v; }
  __device__ __forceinline__ friend Num exp(Num a) { return ::exp(a.v); }
  __device__ __forceinline__ friend Num log(Num a) { return ::log(a.v); }
  __device__ __forceinline__ friend Num sqrt(Num a) { return ::sqrt(a.v); }
  __device__ __forceinline__ friend Num fabs(Num a) { return ::fabs(a.v); }
  __device__ __forceinline__ friend Num pow(Num a, int b) { return ::pow(a.v, b); }
  __device__ __forceinline__ friend Num pow(Num a, double b) { return ::pow(a.v, b); }
  __device__ __forceinline__ friend Num pow(Num a, Num b) { return ::pow(a.v, b.v); }
  __device__ __forceinline__ friend Num pow(double a, Num b) { return ::pow(a, b.v); }
};
__device__ __forceinline__ double value(double x) { return x; }
__device__ __forceinline__ double value(Num x) { return x.v; }

// fmax(fabs(x), fabs(y)) by the bit patterns, off the FP64 pipe.
__device__ __forceinline__ double max_abs(double x, double y) {
  const unsigned long long mask = ~(1ull << 63), inf = 0x7ffull << 52;
  const unsigned long long ax = (unsigned long long)__double_as_longlong(x) & mask;
  const unsigned long long ay = (unsigned long long)__double_as_longlong(y) & mask;
  const bool take_y = ax > inf || (ay <= inf && ay > ax);
  return __longlong_as_double((long long)(take_y ? ay : ax));
}

// ---------------------------------------------------------------------------
// Programs of uniform operations S[out] = fma(+-S[a], S[b], S[c]) or
// S[out] = 1 / S[b], one 64-bit word each, four 16-bit fields of slot * 4 plus
// two flags (emitter/warp_schedule.py):
//   a: 1 negate the product | b, c: 1 the lane's previous result instead |
//   out: 1 store nothing, 2 reciprocal.
// A program with slots beyond 14 bits has words of 128, four 32-bit fields.
// ---------------------------------------------------------------------------
struct alignas(16) WideWord {
  unsigned long long lo, hi;
};
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
  __device__ __forceinline__ unsigned last() const { return hi; }  // the word's end with the out field
};
struct WideProgramWord {
  unsigned fa, fb, fc, fo;
  __device__ __forceinline__ WideProgramWord(const WideWord& w)
      : fa((unsigned)w.lo), fb((unsigned)(w.lo >> 32)), fc((unsigned)w.hi), fo((unsigned)(w.hi >> 32)) {}
  __device__ __forceinline__ unsigned negate() const { return fa << 31; }
  __device__ __forceinline__ bool prev_b() const { return fb & 1u; }
  __device__ __forceinline__ bool prev_c() const { return fc & 1u; }
  __device__ __forceinline__ bool stores() const { return !(fo & 1u); }
  __device__ __forceinline__ bool reciprocal() const { return fo & 2u; }
  __device__ __forceinline__ unsigned a() const { return fa >> 2; }
  __device__ __forceinline__ unsigned b() const { return fb >> 2; }
  __device__ __forceinline__ unsigned c() const { return fc >> 2; }
  __device__ __forceinline__ unsigned out() const { return fo >> 2; }
  __device__ __forceinline__ unsigned last() const { return fo; }
};
__device__ __forceinline__ ProgramWord program_word(unsigned long long w) { return ProgramWord(w); }
__device__ __forceinline__ WideProgramWord program_word(const WideWord& w) { return WideProgramWord(w); }
__device__ __forceinline__ unsigned long long load_word(const unsigned long long* p) { return __ldg(p); }
__device__ __forceinline__ WideWord load_word(const WideWord* p) { return WideWord{__ldg(&p->lo), __ldg(&p->hi)}; }

__device__ __forceinline__ double flip_sign(double x, unsigned sign) {
  return __longlong_as_double(__double_as_longlong(x) ^ ((long long)sign << 32));
}

// Sequential form: one thread runs `ops` words on its own store.  Bound by the
// latency of a word's operands, so those of the next word are loaded before
// this one's result is stored (what it reads of that comes from the register).
// Returns false if a reciprocal met a zero; a program without pivots says so,
// which keeps the division out of its loop.
template <bool kPivots, class SA, class Word>
__device__ __forceinline__ bool run_program(SA& S, const Word* __restrict__ prog, int ops) {
  double prev = 0.0;
  bool ok = true;
  Word now = load_word(prog), next = load_word(prog + (ops > 1 ? 1 : 0));
  double A = S[program_word(now).a()], B = S[program_word(now).b()], C = S[program_word(now).c()];
#pragma unroll 4
  for (int n = 0; n < ops; ++n) {
    const auto w = program_word(now), following = program_word(next);
    now = next;
    next = load_word(prog + (n + 2 < ops ? n + 2 : ops - 1));
    const double a = flip_sign(A, w.negate()), b = w.prev_b() ? prev : B, c = w.prev_c() ? prev : C;
    A = S[following.a()];
    B = S[following.b()];
    C = S[following.c()];
    prev = fma(a, b, c);
    if constexpr (kPivots) {
      if (w.reciprocal()) {
        ok = ok && !is_zero(b);
        prev = divide(1.0, b);
      }
    }
    if (w.stores()) S[w.out()] = prev;
  }
  return ok;
}

}  // namespace mkpp
