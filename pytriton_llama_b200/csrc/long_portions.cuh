// Recurrences that work a portion of many tokens in pieces: which request, and which of its tokens, a piece of the step is.
// Portions of up to `walk_max` tokens have none, a walk over their tokens takes them.  The lengths are read on the device, so
// that a captured step decides by those it is replayed with, and a request's path goes by its own length alone.
#pragma once
#include "common.cuh"

namespace ptl {

// A portion in pieces: its request, first row, tokens, and the number of its first piece among the step's; request -1: there is none.
struct LongPortion { int r, lo, n, piece0; };

// The portion that piece `index` of the step belongs to or, BY_PORTION, the portion of that number (requests in order, pieces
// of PIECE tokens of a request one after the other).  Every warp works it out, 32 requests at a time.
template <bool BY_PORTION, int PIECE>
__device__ __forceinline__ LongPortion locate_portion(const int* __restrict__ q_start, int requests, int walk_max, int index) {
  const int lane = threadIdx.x & 31;
  int pieces_before = 0, portions_before = 0;
  for (int r0 = 0; r0 < requests; r0 += 32) {
    const int r = r0 + lane;
    const int lo = r < requests ? q_start[r] : 0, n = r < requests ? q_start[r + 1] - lo : 0;
    const int pieces = n > walk_max ? (n + PIECE - 1) / PIECE : 0;
    int incl = pieces;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int below = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += below;
    }
    const unsigned with = __ballot_sync(0xffffffffu, pieces > 0);
    const int portion = portions_before + __popc(with & ((1u << lane) - 1u)), piece0 = pieces_before + incl - pieces;
    const unsigned here = __ballot_sync(0xffffffffu, pieces > 0 && (BY_PORTION ? portion == index : index >= piece0 && index < piece0 + pieces));
    if (here) {
      const int who = __ffs(here) - 1;
      return LongPortion{r0 + who, __shfl_sync(0xffffffffu, lo, who), __shfl_sync(0xffffffffu, n, who), __shfl_sync(0xffffffffu, piece0, who)};
    }
    pieces_before += __shfl_sync(0xffffffffu, incl, 31);
    portions_before += __popc(with);
  }
  return LongPortion{-1, 0, 0, 0};
}

}  // namespace ptl
