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


@pytest.mark.parametrize("kind", ["text", "random", "walk", "runs"])
def test_few_chunks(gpu_ctx, oracle_mod, kind):
    """An SM per chunk: more chunks than slots (tables restored between
    them), partial units, one byte, and the same through the pair decoder."""
    data = W.make(kind, 50001, 17).tobytes()
    for unit in (32, 128, 160, 256):
        blob = oracle_mod.compress(data, 5003, unit, 0, 100)
        for tuning in (dict(max_slots=3), dict(max_slots=1), dict(form=cc.FORM_PLAIN), dict(dec_pairs=1)):
            gpu_ctx.set_tuning(**tuning)
            assert gpu_ctx.decompress(blob) == data
    gpu_ctx.set_tuning()
    for n in (1, 2, 15, 16, 17, 33):
        assert gpu_ctx.decompress(oracle_mod.compress(data[:n], 5003, 128, 0, 100)) == data[:n]


@pytest.mark.parametrize("chunks", [63, 64, 65, 149])
def test_around_the_switch(gpu_ctx, oracle_mod, chunks):
    gpu_ctx.set_tuning()
    data = W.text(chunks * 700 - 3, chunks).tobytes()
    assert gpu_ctx.decompress(oracle_mod.compress(data, 700, 128, 0, 100)) == data


def test_prelearned_few_chunks(gpu_ctx, oracle_mod):
    gpu_ctx.set_tuning(max_slots=2)
    data = W.text(60000, 4).tobytes()
    assert gpu_ctx.decompress(oracle_mod.compress(data, 8000, 128, 9000, 100)) == data
    gpu_ctx.set_tuning()


@pytest.mark.parametrize("pairs", [0, 1, 2])
def test_waits_that_run_out(gpu_ctx, oracle_mod, pairs):
    data = W.text(100_000, 21).tobytes()
    blob = oracle_mod.compress(data, 20000, 128, 0, 100)
    gpu_ctx.set_tuning(dec_pairs=pairs, dec_spin_limit=1)
    with pytest.raises(cc.CucmError) as e:
        gpu_ctx.decompress(blob)
    assert e.value.status == -7
    gpu_ctx.set_tuning(dec_pairs=pairs)
    assert gpu_ctx.decompress(blob) == data
    gpu_ctx.set_tuning()
