// warp_wait.h -- a bounded wait that a warp's lanes leave together.
//
// What follows a wait is warp-wide (shuffles, votes, named barriers), so a lane
// that saw the word in time must not part from one that did not: the lanes vote,
// and the outcome is the warp's.  Lanes that poll for themselves agree only while
// they happen to run in step.  One vote at the end; one with every poll made the
// decoder with an SM per chunk 1.2 % slower.
#pragma once

#include <cstdint>

#ifndef __CUDACC__
#define CUCM_WAIT_FN inline
#else
#define CUCM_WAIT_FN __device__ __forceinline__
#endif

namespace cucm {

// Each lane polls until its there() holds, `limit` times at most (at least once);
// whether all saw it.  all(x): whether x holds in every lane of the warp.  then():
// what a lane does before the vote is in, whatever its outcome.
template <class There, class All, class Then>
CUCM_WAIT_FN bool warp_wait(There there, All all, uint32_t limit, Then then) {
  bool seen = there();
  for (uint32_t polls = 1; !seen && polls < limit; polls++) seen = there();
  then();
  return all(seen);
}

}  // namespace cucm
