"""Waits of the decoder with an SM per chunk that run out at some bytes and not
at others: the call ends with the data or with the timeout, and the context
decodes on."""
import pytest

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu

ETIMEOUT = -7


@pytest.mark.parametrize("limit", [1, 2, 16, 64, 256, 1024])
@pytest.mark.parametrize("unit", [32, 256])
def test_waits_that_run_out_on_the_way(gpu_ctx, oracle_mod, limit, unit):
    data = b"".join(W.make(kind, 6000, limit).tobytes() for kind in ("text", "random", "runs", "walk"))
    blob = oracle_mod.compress(data, 3001, unit, 0, 100)
    gpu_ctx.set_tuning(dec_spin_limit=limit)
    try:
        assert gpu_ctx.decompress(blob) == data
    except cc.CucmError as e:
        assert e.status == ETIMEOUT
    gpu_ctx.set_tuning()
    assert gpu_ctx.decompress(blob) == data
