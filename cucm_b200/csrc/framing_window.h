// framing_window.h -- a container's framing read piece by piece from memory
// that costs a blocking copy to read.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace cucm {

// Batches' size fields and tables lie payloads apart and are read front to
// back.  A copy takes ~10 us before its first byte, in which pageable memory
// takes ~15 KB of a long one, so where the next batch begins less than
// kFramingGap behind the piece at hand the payloads between are not worth
// leaving out: pieces grow until the container comes in long ones.  Where it
// begins further on, a piece holds just its framing.  Calls of 4,000 batches of
// one 256-byte chunk: 231 ms with the container in one copy, 324 with two copies
// a batch, 229 so; of 2,000 batches 12 KB apart 297, 387 and 293.
constexpr uint64_t kFramingPiece = 4096;      // tables of up to ~1,000 chunks
constexpr uint64_t kFramingGap = 32 << 10;
constexpr uint64_t kFramingMost = 1 << 20;

// fetch(at, n, dst) copies n bytes from offset `at` and returns whether it could.
template <class Fetch>
class FramingWindow {
 public:
  // `from`: where the framing goes on behind what the caller holds already.
  FramingWindow(Fetch fetch, uint64_t total, uint64_t from) : fetch_(fetch), total_(total), at_(from) {}

  // n bytes from offset `at` (at + n <= total), or null when a copy failed.
  const uint8_t *read(uint64_t at, uint64_t n) {
    const uint64_t end = at_ + buf_.size();
    if (at < at_ || at + n > end) {
      const bool near = at + n >= end && at <= end + kFramingGap;
      piece_ = near ? std::min(8 * piece_, kFramingMost) : kFramingPiece;
      buf_.resize(std::min(std::max(n, piece_), total_ - at));
      at_ = at;
      if (!fetch_(at, buf_.size(), buf_.data())) return nullptr;
    }
    return buf_.data() + (at - at_);
  }

 private:
  Fetch fetch_;
  uint64_t total_, at_;
  uint64_t piece_ = kFramingPiece;
  std::vector<uint8_t> buf_;
};

}  // namespace cucm
