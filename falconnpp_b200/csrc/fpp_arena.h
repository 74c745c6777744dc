// fpp_arena.h — reservation of ranges of different lengths from one counter by
// many threads at once (the put-off tie repairs of fpp_build.cu).
#pragma once

#if defined(__CUDACC__)
#define FPP_ARENA_HD __host__ __device__ __forceinline__
#else
#define FPP_ARENA_HD inline
#endif

namespace fpp {

constexpr unsigned kArenaFull = 0xffffffffu;

// The start of `want` units out of `cap`, or kArenaFull.  load() reads the
// counter, cas(expect, value) is a compare-and-swap that returns what was
// there.  The counter moves only by reservations that hold, so it never goes
// back below a range handed out (an add that a failing thread takes back
// afterwards lets a shorter range in above itself, and the subtraction then
// hands that range out twice), and it never passes `cap`.
template <typename Load, typename Cas>
FPP_ARENA_HD unsigned arena_reserve(unsigned want, unsigned cap, Load load, Cas cas) {
  unsigned cur = load();
  while (cur <= cap && want <= cap - cur) {
    const unsigned was = cas(cur, cur + want);
    if (was == cur) return cur;
    cur = was;
  }
  return kArenaFull;
}

}  // namespace fpp
