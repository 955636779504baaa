"""The coder's groups of 16 bits: bits that shift out several bytes at once,
units and tails that are no multiple of a group, and more chunks than the
device has warp schedulers (several chunks to a warp of the tail pass and of
the fixed-model coder).  Containers equal the oracle's byte for byte."""
import numpy as np
import pytest

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _surprises(n, every, seed):
    """Long runs of one byte broken by random ones: bits coded against odds
    of up to 2^12."""
    rng = np.random.default_rng(seed)
    out = np.full(n, 0x20, dtype=np.uint8)
    at = np.arange(every, n, every)
    out[at] = rng.integers(0, 256, size=at.size, dtype=np.uint8)
    return out


@pytest.mark.parametrize("n,cs,unit", [(30000, 8192, 128), (30000, 8191, 32), (9999, 20003, 256), (5000, 5001, 96),
                                       (4097, 9000, 160)])
@pytest.mark.parametrize("every", [37, 1000])
def test_surprises(gpu_ctx, oracle_mod, n, cs, unit, every):
    data = _surprises(n, every, n + every).tobytes()
    want = oracle_mod.compress(data, cs, unit, 0, 100)
    for kernel in (0, 1):
        for form in (cc.FORM_PERSISTENT, cc.FORM_PLAIN):
            gpu_ctx.set_tuning(form=form, kernel=kernel)
            assert gpu_ctx.compress(data, cs, unit) == want


@pytest.mark.parametrize("count", [593, 1300])  # 2 and 4 chunks to a warp with 148 SMs
def test_many_tails(gpu_ctx, oracle_mod, count):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT)
    bufs = [(_surprises(20 + i % 90, 7, i) if i % 3 else W.make("text", 20 + i % 90, i)).tobytes()
            for i in range(count)]
    got = gpu_ctx.compress_many(bufs, chunksize=1000 + 7)
    for i in range(0, count, 41):
        assert got[i] == oracle_mod.compress(bufs[i], 1007, 128, 0, 100)
    assert gpu_ctx.decompress_many(got) == bufs


def test_many_fixed_chunks(gpu_ctx, oracle_mod):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT)
    data = np.concatenate([W.text(40000, 5), _surprises(120001, 50, 6)]).tobytes()
    want = oracle_mod.compress(data, 111, 128, 20000, 100, fixed=True)  # 1,262 chunks of an odd size
    assert gpu_ctx.compress(data, 111, 128, 20000, 100, fixed=True) == want
    assert gpu_ctx.decompress(want) == data
