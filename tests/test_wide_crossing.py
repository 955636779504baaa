"""How the wide decoder's warps cross a byte when the decoding warp's wait for a
prediction runs out: every interleaving of the decoding warp and two guessing
warps, with the number of barriers and byte places that the kernels use."""
import os
import subprocess

import pytest

import cucm_b200 as cc

CSRC = os.path.join(os.path.dirname(os.path.abspath(cc.__file__)), "csrc")
BYTES = 5


@pytest.fixture(scope="module")
def used(tmp_path_factory):
    """(barriers, places) of the kernels' header."""
    d = tmp_path_factory.mktemp("crossing")
    src, exe = d / "m.cpp", d / "m"
    src.write_text('#include <cstdio>\n#include "wide_crossing.h"\n'
                   'int main() { std::printf("%u %u", cucm::kWideBarriers, cucm::kWidePlaces); }\n')
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    return tuple(int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())


def _explore(barriers, places, path, recovers):
    """Faults that some interleaving meets.  path[n]: the guessing warp whose
    prediction byte n needs.  recovers: a byte after one whose wait ran out may
    arrive again (the fixed-model decoder).

    Decoding warp: (0 waits for path[n]'s prediction, 1 writes byte n, 2 comes to
    crossing n, 3 waits in it; n; ok).  Guessing warp: (0 publishes its prediction
    of byte n, 1 comes to crossing n, 2 waits in it, 3 reads byte n; n)."""
    warps = max(path) + 1
    start = ((0, 0, True), ((0, 0),) * warps, (0,) * warps, ((),) * barriers, (-1,) * places)
    seen, todo, faults = {start}, [start], set()

    def put(t, i, v):
        return t[:i] + (v,) + t[i + 1:]

    def arrive(who, n, dec, gs, bars):
        b = n % barriers
        here = bars[b] + (who,)
        if here.count(who) > 1:
            faults.add("counted twice")
        if len(here) < warps + 1:
            return dec, gs, put(bars, b, here)
        for w in here:
            if w >= 0 and gs[w][0] == 2:
                gs = put(gs, w, (3, gs[w][1]))
            elif w < 0 and dec[0] == 3:
                dec = (0, dec[1] + 1, recovers)
        return dec, gs, put(bars, b, ())

    while todo:
        dec, gs, ready, bars, place = todo.pop()
        pc, n, ok = dec
        after = []
        if n < BYTES:
            if pc == 0:
                if ready[path[n]] > n and ok:
                    after.append(((1, n, True), gs, ready, bars, place))
                else:
                    after.append(((1, n, False), gs, ready, bars, place))
            elif pc == 1:
                after.append(((2, n, ok), gs, ready, bars, put(place, n % places, n)))
            elif pc == 2:
                d, g, b = arrive(-1, n, (0, n + 1, ok) if ok else (3, n, ok), gs, bars)
                after.append((d, g, ready, b, place))
        for w, (gpc, m) in enumerate(gs):
            if m >= BYTES:
                continue
            if gpc == 0:
                after.append((dec, put(gs, w, (1, m)), put(ready, w, m + 1), bars, place))
            elif gpc == 1:
                d, g, b = arrive(w, m, dec, put(gs, w, (2, m)), bars)
                after.append((d, g, ready, b, place))
            elif gpc == 3:
                if place[m % places] != m:
                    faults.add("wrong byte")
                after.append((dec, put(gs, w, (0, m + 1)), ready, bars, place))
        if not after and not (n >= BYTES and all(m >= BYTES for _, m in gs)):
            faults.add("never meets again")
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return faults


@pytest.mark.parametrize("recovers", [False, True], ids=["adaptive", "fixed"])
@pytest.mark.parametrize("path", [(0, 1, 0, 1, 0), (1, 1, 1, 1, 1), (1, 0, 0, 1, 1)])
def test_every_interleaving_meets(used, path, recovers):
    assert _explore(*used, path, recovers) == set()


def test_the_search_sees_the_faults():
    path = (0, 1, 0, 1, 0)
    assert {"counted twice", "never meets again"} <= _explore(1, 4, path, False)
    assert _explore(2, 2, path, False) == {"wrong byte"}
