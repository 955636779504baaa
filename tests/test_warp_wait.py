"""A bounded wait's outcome is the warp's: whatever lane sees the word in time and
whatever lane does not, all leave with the same answer."""
import itertools
import os
import subprocess

import pytest

import cucm_b200 as cc

CSRC = os.path.join(os.path.dirname(os.path.abspath(cc.__file__)), "csrc")
LANES, LIMIT = 3, 4

# Each lane runs on a thread of its own; a vote is a rendezvous of all lanes.  The
# lane's k-th poll (from 0) sees the word from k = seen[lane] on.
SOURCE = r"""
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
#include "warp_wait.h"
struct Votes {
  std::mutex m;
  std::condition_variable cv;
  int lanes, in = 0, round = 0;
  bool all = true, last = true;
  bool vote(bool x) {
    std::unique_lock<std::mutex> g(m);
    const int r = round;
    all = all && x;
    if (++in == lanes) {
      last = all;
      all = true;
      in = 0;
      round++;
      cv.notify_all();
    } else {
      cv.wait(g, [&] { return round != r; });
    }
    return last;
  }
};
int main(int n, char **v) {  // limit, seen...
  const uint32_t limit = (uint32_t)atoi(v[1]);
  Votes votes;
  votes.lanes = n - 2;
  std::vector<int> got(n - 2), polls(n - 2);
  std::vector<std::thread> t;
  for (int i = 0; i < n - 2; i++)
    t.emplace_back([&, i] {
      got[i] = cucm::warp_wait([&] { return polls[i]++ >= atoi(v[2 + i]); }, [&](bool x) { return votes.vote(x); }, limit, [] {});
    });
  for (auto &x : t) x.join();
  for (int i = 0; i < n - 2; i++) std::printf("%d/%d ", got[i], polls[i]);
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + CSRC, str(d / "m.cpp"), "-o", str(d / "m")],
                   check=True)
    return str(d / "m")


def test_lanes_leave_together(exe):
    for limit in (1, LIMIT):
        for seen in itertools.product(range(LIMIT + 2), repeat=LANES):
            out = subprocess.run([exe, str(limit)] + [str(x) for x in seen], capture_output=True, text=True,
                                 check=True, timeout=60).stdout.split()
            there = max(seen) < limit  # the last lane's sight decides
            assert out == ["%d/%d" % (there, min(k + 1, limit)) for k in seen]


def test_the_decoders_wait_through_it():
    """No wait of the decoders that a lane could leave by itself."""
    for name in ("decompress_fast.cuh", "decompress_wide.cuh"):
        text = open(os.path.join(CSRC, name)).read()
        assert "dec_wait(" in text and "spins" not in text
