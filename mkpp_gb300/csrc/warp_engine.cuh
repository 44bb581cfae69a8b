// Runs the warp-cooperative programs (emitter/warp_schedule.py; word layout in
// mkpp_device.cuh).
#pragma once
#include <type_traits>

#include "mkpp_device.cuh"

namespace mkpp {

constexpr int kProgramAhead = 8;

// What the loop below takes from the words of a program: the byte offsets of
// the slots, and how the words of a group of steps lie in memory.
template <class Word>
struct StepWords;

// 64-bit words, two steps' words of a lane side by side.  A field (slot * 4 +
// flags), shifted to slot * 8, is a byte offset.
template <>
struct StepWords<unsigned long long> {
  typedef unsigned long long Word;
  static constexpr unsigned kIdle = 0x10000u;  // last field and its half word: nothing to store
  __device__ __forceinline__ static void fetch(const ulonglong2* __restrict__ words, int g, Word* to) {
    constexpr int kPairs = kProgramAhead / 2;
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      const ulonglong2 v = __ldg(words + ((size_t)g * kPairs + j) * 32);
      to[2 * j] = v.x;
      to[2 * j + 1] = v.y;
    }
  }
  __device__ __forceinline__ static unsigned a(Word v) { return ((unsigned)v << 1) & 0x1fff8u; }
  __device__ __forceinline__ static unsigned b(Word v) { return ((unsigned)v >> 15) & 0x1fff8u; }
  __device__ __forceinline__ static unsigned c(Word v) { return ((unsigned)(v >> 32) << 1) & 0x1fff8u; }
  __device__ __forceinline__ static unsigned last(Word v) { return (unsigned)(v >> 32); }
  __device__ __forceinline__ static unsigned out(unsigned last) { return (last >> 15) & 0x1fff8u; }
  __device__ __forceinline__ static bool stores(unsigned last) { return !(last & 0x10000u); }
  __device__ __forceinline__ static bool reciprocal(unsigned last) { return last & 0x20000u; }
};

// 128-bit words.
template <>
struct StepWords<WideWord> {
  static constexpr unsigned kIdle = 1u;
  __device__ __forceinline__ static void fetch(const ulonglong2* __restrict__ words, int g, WideWord* to) {
#pragma unroll
    for (int j = 0; j < kProgramAhead; ++j) {
      const ulonglong2 v = __ldg(words + ((size_t)g * kProgramAhead + j) * 32);
      to[j] = WideWord{v.x, v.y};
    }
  }
  __device__ __forceinline__ static unsigned a(const WideWord& v) { return WideProgramWord(v).a() * 8u; }
  __device__ __forceinline__ static unsigned b(const WideWord& v) { return WideProgramWord(v).b() * 8u; }
  __device__ __forceinline__ static unsigned c(const WideWord& v) { return WideProgramWord(v).c() * 8u; }
  __device__ __forceinline__ static unsigned last(const WideWord& v) { return (unsigned)(v.hi >> 32); }
  __device__ __forceinline__ static unsigned out(unsigned last) { return (last >> 2) * 8u; }
  __device__ __forceinline__ static bool stores(unsigned last) { return !(last & 1u); }
  __device__ __forceinline__ static bool reciprocal(unsigned last) { return last & 2u; }
};

// One warp runs `steps` steps (a multiple of kProgramAhead, the last one idle)
// of 32 words, a lane per word, on one store that the warp shares; reciprocals
// only in the last of kPivotEvery steps.
//
// Bound by latency: a GB300 warp issues one FP64 instruction per 64 cycles,
// whatever its active lanes, and an FMA whose result anything but the next FMA
// uses takes 108, so a step is an FMA, the store of its result and the loads of
// the next operands.  Measured on SAPRC99's 2296 steps, up to four warps on an SM:
// 164 cycles a step in the LU (5 of them bank conflicts, some 28 the steps with
// reciprocals, by their number) and 111-120 in the solves, and with eight 209 and
// 143-150 (the FP64 pipe's bound there is 138: 2482 instructions an attempt, two
// warps to a pipe); 172 and 204 on average with a vote for pivots in every
// step, operand loads under branches and the words of a step each waited for
// alone.
template <int kPivotEvery>
struct WarpProgram {
  // Returns false if a reciprocal of this lane met a zero.
  template <class Word>
  __device__ __forceinline__ bool operator()(double* S, const Word* __restrict__ prog, int steps, unsigned lane) const {
    typedef StepWords<Word> Words;
    const ulonglong2* __restrict__ words = reinterpret_cast<const ulonglong2*>(prog) + lane;
    char* const base = reinterpret_cast<char*>(S);
    const int groups = steps / kProgramAhead;
    Word w[kProgramAhead];
    auto at = [&](unsigned offset) { return reinterpret_cast<double*>(base + offset); };
    double A, B, C, prev = 0.0;
    auto load = [&](Word v) {
      A = flip_sign(*at(Words::a(v)), program_word(v).negate());
      B = *at(Words::b(v));
      C = *at(Words::c(v));
    };
    unsigned before = Words::kIdle;  // the previous step's last field: nothing to store yet
    bool ok = true;
    // One group of steps; only some groups hold pivots.
    auto run = [&](auto pivots, Word first_after) {
#pragma unroll
      for (int j = 0; j < kProgramAhead; ++j) {
        const auto p = program_word(w[j]);
        const double b = p.prev_b() ? prev : B;
        const double c = p.prev_c() ? prev : C;
        double v = fma(A, b, c);
        if (decltype(pivots)::value && j % kPivotEvery == kPivotEvery - 1) {
          if (__any_sync(0xffffffffu, p.reciprocal())) {
            ok = ok && !(p.reciprocal() && is_zero(b));
            const double r = divide(1.0, p.reciprocal() ? b : 1.0);
            v = p.reciprocal() ? r : v;
          }
        }
        if (Words::stores(before)) *at(Words::out(before)) = prev;
        __syncwarp();
        load(j + 1 < kProgramAhead ? w[j + 1] : first_after);
        prev = v;
        before = p.last();
      }
    };
    Words::fetch(words, 0, w);
    load(w[0]);
    for (int g = 0; g < groups; ++g) {
      Word next[kProgramAhead];
      Words::fetch(words, g + 1 < groups ? g + 1 : g, next);
      unsigned any = 0;
#pragma unroll
      for (int j = 0; j < kProgramAhead; ++j) any |= Words::last(w[j]);
      if (__any_sync(0xffffffffu, Words::reciprocal(any)))
        run(std::true_type(), next[0]);
      else
        run(std::false_type(), next[0]);
#pragma unroll
      for (int j = 0; j < kProgramAhead; ++j) w[j] = next[j];
    }
    if (Words::stores(before)) *at(Words::out(before)) = prev;
    __syncwarp();
    return ok;
  }
};

}  // namespace mkpp
