"""Reading a container's framing from device memory: what the batch parser asks
for arrives whole, in a number of copies that the batches' spacing does not
multiply."""
import os
import subprocess

import pytest

import cucm_b200 as cc

CSRC = os.path.join(os.path.dirname(os.path.abspath(cc.__file__)), "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "framing_window.h"
// argv: container bytes, bytes held, first batch, batch spacing, framing bytes of a batch, copy that fails
int main(int, char **v) {
  const uint64_t total = strtoull(v[1], 0, 0), held = strtoull(v[2], 0, 0), first = strtoull(v[3], 0, 0),
                 step = strtoull(v[4], 0, 0), need = strtoull(v[5], 0, 0);
  const long bad = strtol(v[6], 0, 0);
  auto byte = [](uint64_t i) { return (uint8_t)(i * 2654435761u >> 13); };
  uint64_t copies = 0, bytes = 0, reads = 0;
  auto fetch = [&](uint64_t at, uint64_t n, uint8_t *to) {
    if (at + n > total) exit(2);
    if ((long)copies++ == bad) return false;
    bytes += n;
    for (uint64_t i = 0; i < n; i++) to[i] = byte(at + i);
    return true;
  };
  cucm::FramingWindow<decltype(fetch)> w(fetch, total, held);
  for (uint64_t at = first; at < total; at += step, reads++) {
    const uint64_t n = std::min(need, total - at);
    for (uint64_t o = 0; o <= 4; o += 4) {  // the size field with its table, then the table
      if (n < o + 1 || at + n <= held) continue;
      const uint8_t *p = w.read(at + o, n - o);
      if (!p) return std::printf("failed"), 0;
      for (uint64_t i = 0; i < n - o; i++)
        if (p[i] != byte(at + o + i)) exit(3);
    }
  }
  std::printf("%llu %llu %llu", (unsigned long long)reads, (unsigned long long)copies, (unsigned long long)bytes);
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("framing")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, str(d / "m.cpp"), "-o", str(d / "m")], check=True)
    return str(d / "m")


def _run(exe, *args):
    return subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, check=True).stdout


@pytest.mark.parametrize("need", [8, 404, 5000, 70000])
@pytest.mark.parametrize("spacing", [1, 100, 4095, 4097, 20000, 32768, 40000, 66000, 1 << 20])
def test_copies(exe, need, spacing):
    total, held = 12345678, 4096
    spacing += need
    for first in (45, 4000, 9000):
        reads, copies, copied = (int(x) for x in _run(exe, total, held, first, spacing, need, -1).split())
        assert reads == (total - first + spacing - 1) // spacing
        assert copies <= reads
        # a copy costs what ~15 KB of a long one do; the whole in one copy is the measure
        assert copied + 15000 * copies <= 1.25 * total + 200000


def test_a_copy_that_fails(exe):
    for bad in (0, 1, 50):
        assert _run(exe, 8 << 20, 4096, 45, 100000, 8, bad) == "failed"
