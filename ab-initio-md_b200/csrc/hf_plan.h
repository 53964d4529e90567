// How a context's launch shape (aimd_set_launch_shape) sets the work plan of a
// class launch: the number of chunks it is cut into, and the length of its
// split column items. Plain C++, for the planner on both sides.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define AIMD_HD __host__ __device__
#else
#define AIMD_HD
#endif

namespace hf {

constexpr int DEFAULT_CHUNKS = 8, DEFAULT_ITEM_PQ = 32;

// Chunks that the work of a launch is cut into (bras of little work are one
// chunk each all the same). At the default per_sm an SM; any other value is
// taken literally, two CTAs an SM. per_sm is 2 for J/K and 4 for the gradient:
// with 16, as many as the bras of a large molecule make anyway, (H2O)32 J/K
// took 79 against 73 ms and the (H2O)8 difference build 5.6 against 2.8, in one
// CTA an SM.
AIMD_HD inline int plan_parts(int chunks, int per_sm, int nsm) {
    return (chunks == DEFAULT_CHUNKS ? per_sm : 2 * chunks) * nsm;
}

// Primitive quartets of a split item in a launch of W work units (a unit is half
// a primitive quartet of a column) on a device of `threads` threads. At the
// default at most that many, and fewer where the launch would not give two items
// to each thread; any other value is taken literally. Launches of little work
// are bound by their longest item, a chain of primitive quartets in one thread:
// shorter ones took the build of a UHF molecule of 24 functions from 550 to
// 473 us and the gradient of methanol from 696 to 669, where items of 4 instead
// of 32 quartets everywhere cost the large launches a digest each.
constexpr int MIN_ITEM_PQ = 4;
AIMD_HD inline int split_length(int64_t W, int item_pq, int threads) {
    if (item_pq != DEFAULT_ITEM_PQ) return item_pq;
    const int64_t even = W / (4 * (int64_t)threads);
    return even >= item_pq ? item_pq : (even < MIN_ITEM_PQ ? MIN_ITEM_PQ : static_cast<int>(even));
}

}  // namespace hf
