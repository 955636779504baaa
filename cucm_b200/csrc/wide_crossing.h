// wide_crossing.h -- what the decoders with an SM per chunk cross a byte with.
//
// Named barriers 1 and up (0 is the CTA's), in turn by byte: byte n is known.
// The decoding warp arrives and goes on, the guessing warps wait, then read the
// byte.
//
// The decoding warp leaves byte n in one of two ways.  It has seen a `ready` of
// byte n, whose writer came through crossing n - 1 with all the others, and
// arrives.  Or its wait for that `ready` has run out, so that crossing n - 1 may
// still be open, and it waits at crossing n until the guessing warps have come
// through both.  Either way crossing n - 1 is complete when it reaches crossing
// n + 1; with two barriers that is the next one to use the same barrier, so the
// warp is never counted twice in one crossing.  (With one barrier the second way
// is: the crossing closes without a warp that is late, which then stays one
// behind, and the CTA never meets again.)
//
// When the decoding warp writes byte n, all guessing warps have come to crossing
// n - 2 (crossing n - 1 in the first way) and so have read byte n - 3, but one may
// still have to read byte n - 2: three places, or four to index with a mask.
#pragma once

#include <cstdint>

namespace cucm {

constexpr uint32_t kWideBarriers = 2;
constexpr uint32_t kWidePlaces = 4;

}  // namespace cucm
