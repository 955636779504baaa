"""The 8 keys of a byte and an order never meet, in the code that makes them
(model.cuh): the compressor's walker and the decoder's updater take a byte's or a
nibble's bits together on the strength of it."""
import os
import subprocess

import pytest

import cucm_b200 as cc

CSRC = os.path.join(os.path.dirname(os.path.abspath(cc.__file__)), "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "model.cuh"
// partial bytes of one history and order that share a slot, over many histories
int main() {
  using namespace cucm;
  uint32_t rnd = 12345;
  auto next = [&] { return (rnd = rnd * 1664525u + 1013904223u) >> 24; };
  static int owner[kSlotTableBytes];  // history number of the slot's last key
  long long meets = 0;
  for (int n = 1; n <= 3000; n++) {
    uint32_t hist[7];
    for (uint32_t &h : hist) h = n % 3 == 0 ? (next() & 1u) * 255u : next();
    for (uint32_t h0 = 1; h0 < 256; h0++) {
      BitKeys k;
      bit_keys(h0, hist, k);
      for (int o = 0; o < kOrders; o++) {
        const uint64_t end = o + 1 < kOrders ? table_offset(o + 1) : kSlotTableBytes, at = table_offset(o) + k.k[o];
        if (at >= end) return 2;
        meets += owner[at] == n;
        owner[at] = n;
      }
    }
  }
  std::printf("%lld", meets);
}
"""


def _meets(d, change=lambda text: text):
    text = open(os.path.join(CSRC, "model.cuh")).read()
    (d / "model.cuh").write_text(change(text))
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-D__host__=", "-D__device__=", "-I" + str(d), str(d / "m.cpp"),
                    "-o", str(d / "m")], check=True)
    return int(subprocess.run([str(d / "m")], capture_output=True, text=True, check=True).stdout)


def test_partial_bytes_never_meet(tmp_path):
    assert _meets(tmp_path) == 0


@pytest.mark.parametrize("old,new", [("kFnvPrime = 16777619u", "kFnvPrime = 16777616u"),
                                     ("out.k[o] = acc & (kSlots - 1)", "out.k[o] = acc & (kSlots - 1) & ~4u")])
def test_a_hash_that_is_not_one_to_one_is_seen(tmp_path, old, new):
    def change(text):
        assert text.count(old) == 1
        return text.replace(old, new)
    assert _meets(tmp_path, change) > 0
