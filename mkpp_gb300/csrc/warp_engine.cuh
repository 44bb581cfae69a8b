// Runs the warp-cooperative programs (emitter/warp_schedule.py; word layout in
// mkpp_device.cuh).
#pragma once
#include <type_traits>

#include "mkpp_device.cuh"

namespace mkpp {

constexpr int kProgramAhead = 8;

// One warp runs `steps` steps (a multiple of kProgramAhead, the last one idle)
// of 32 words, a lane per word, two steps' words of a lane side by side, on
// one store that the warp shares; reciprocals only in the last of kPivotEvery
// steps.
//
// Bound by latency: a GB300 warp issues one FP64 instruction per 64 cycles,
// whatever its active lanes, and an FMA whose result anything but the next FMA
// uses takes 108, so a step is an FMA, the store of its result and the loads of
// the next operands.  Measured on SAPRC99's 2296 steps, up to four warps on an SM:
// 164 cycles a step in the LU (5 of them bank conflicts, some 28 the steps with
// reciprocals, by their number) and 111-120 in the solves, and with eight 209 and 143-150 (the FP64 pipe's
// bound there is 152); 172 and 204 on average with a vote for pivots in every
// step, operand loads under branches and the words of a step each waited for
// alone.
template <int kPivotEvery>
struct WarpProgram {
  // Returns false if a reciprocal of this lane met a zero.
  __device__ __forceinline__ bool operator()(double* S, const unsigned long long* __restrict__ prog, int steps,
                                             unsigned lane) const {
    constexpr int kPairs = kProgramAhead / 2;
    const ulonglong2* __restrict__ words = reinterpret_cast<const ulonglong2*>(prog) + lane;
    char* const base = reinterpret_cast<char*>(S);
    const int groups = steps / kProgramAhead;
    unsigned long long w[kProgramAhead];
    auto fetch = [&](int g, unsigned long long* to) {
#pragma unroll
      for (int j = 0; j < kPairs; ++j) {
        const ulonglong2 v = __ldg(words + ((size_t)g * kPairs + j) * 32);
        to[2 * j] = v.x;
        to[2 * j + 1] = v.y;
      }
    };
    // A field (slot * 4 + flags), shifted to slot * 8, is its byte offset.
    auto at = [&](unsigned offset) { return reinterpret_cast<double*>(base + (offset & 0x1fff8u)); };
    double A, B, C, prev = 0.0;
    auto load = [&](unsigned long long v) {
      const unsigned lo = (unsigned)v, hi = (unsigned)(v >> 32);
      A = flip_sign(*at(lo << 1), lo << 31);
      B = *at(lo >> 15);
      C = *at(hi << 1);
    };
    unsigned before = 0x10000u;  // the previous step's high word: nothing to store yet
    bool ok = true;
    // One group of steps; only some groups hold pivots.
    auto run = [&](auto pivots, unsigned long long first_after) {
#pragma unroll
      for (int j = 0; j < kProgramAhead; ++j) {
        const ProgramWord p(w[j]);
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
        if (!(before & 0x10000u)) *at(before >> 15) = prev;
        __syncwarp();
        load(j + 1 < kProgramAhead ? w[j + 1] : first_after);
        prev = v;
        before = p.hi;
      }
    };
    fetch(0, w);
    load(w[0]);
    for (int g = 0; g < groups; ++g) {
      unsigned long long next[kProgramAhead];
      fetch(g + 1 < groups ? g + 1 : g, next);
      unsigned any = 0;
#pragma unroll
      for (int j = 0; j < kProgramAhead; ++j) any |= (unsigned)(w[j] >> 32);
      if (__any_sync(0xffffffffu, any & 0x20000u))
        run(std::true_type(), next[0]);
      else
        run(std::false_type(), next[0]);
#pragma unroll
      for (int j = 0; j < kProgramAhead; ++j) w[j] = next[j];
    }
    if (!(before & 0x10000u)) *at(before >> 15) = prev;
    __syncwarp();
    return ok;
  }
};

}  // namespace mkpp
