"""The decoder's round: bits that shift several payload bytes at once
(odds of up to 2^12), slots that recur within a unit and across units (the
updating warp's position hash), states met several times in a nibble, and
payloads that end on every byte of a 16-byte block."""
import numpy as np
import pytest

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _surprises(n, every, seed):
    rng = np.random.default_rng(seed)
    out = np.full(n, 0x20, dtype=np.uint8)
    at = np.arange(every, n, every)
    out[at] = rng.integers(0, 256, size=at.size, dtype=np.uint8)
    return out


@pytest.mark.parametrize("unit", [32, 128, 256])
@pytest.mark.parametrize("every", [3, 37, 1000])
@pytest.mark.parametrize("tables", [0, 1], ids=["shared", "slot"])
def test_rounds(gpu_ctx, oracle_mod, unit, every, tables):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT, dec_tables=tables)
    data = _surprises(40000, every, every + unit).tobytes()
    for cs in (40000, 7777, 512):
        blob = oracle_mod.compress(data, cs, unit, 0, 100)
        assert gpu_ctx.decompress(blob) == data
    gpu_ctx.set_tuning()


@pytest.mark.parametrize("kind", ["text", "random", "runs"])
def test_short_payloads(gpu_ctx, oracle_mod, kind):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT)
    bufs = [W.make(kind, n, n).tobytes() for n in range(1, 70)]
    blobs = [oracle_mod.compress(b, 70, 64, 0, 100) for b in bufs]
    assert gpu_ctx.decompress_many(blobs) == bufs
    whole = b"".join(bufs)  # 70-byte chunks one after the other: every payload offset mod 16
    assert gpu_ctx.decompress(oracle_mod.compress(whole, 70, 64, 0, 100)) == whole


@pytest.mark.parametrize("pairs", [1, 2, 3, 5])
def test_pairs_per_cta(gpu_ctx, oracle_mod, pairs):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT, dec_pairs=pairs)
    data = W.text(60000, 9).tobytes()
    for unit in (96, 224):
        blob = oracle_mod.compress(data, 5000, unit, 0, 100)
        assert gpu_ctx.decompress(blob) == data
    gpu_ctx.set_tuning()
