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
// counter, add(v) adds to it and returns what was there.  The counter never
// goes back (an add that a failing thread takes back afterwards lets a shorter
// range in above itself, and the subtraction then hands that range out twice):
// a reservation that loses a race near the end leaves it past `cap`, what was
// left stays unused, and later callers no longer add.  So it ends at most one
// failed range per thread past `cap`, whose sum the caller keeps below 2^32.
// (A compare-and-swap loop wastes nothing, but every success is a round trip to
// L2 after the last one: 1 us each, 65,000 tied buckets 128 ms.)
template <typename Load, typename Add>
FPP_ARENA_HD unsigned arena_reserve(unsigned want, unsigned cap, Load load, Add add) {
  const unsigned cur = load();
  if (cur > cap || want > cap - cur) return kArenaFull;
  const unsigned pos = add(want);
  return pos <= cap && want <= cap - pos ? pos : kArenaFull;
}

}  // namespace fpp
