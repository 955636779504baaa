"""Autotuner candidates that come to the same launch are one choice: they share a
time, and the derived rule's name is the one that is applied."""
import pytest
import torch

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx(gpu_ctx):
    yield gpu_ctx
    gpu_ctx.set_tuning()


def _times(cands, field, form):
    return {(c["cmp_ctas"], c["dec_pairs"], c["dec_tables"]): c[field] for c in cands
            if c["form"] == form and c["kernel"] == 0 and c[field] >= 0}


@pytest.mark.parametrize("more", [16, 2 * 148 + 5])
def test_one_launch_has_one_time(ctx, more):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chunks = more if more < sms else 2 * sms + 5
    best, cands = ctx.autotune(W.make("text", 1024 * chunks, 3).tobytes(), reps=1, chunksize=1024)
    comp = _times(cands, "compress_ms", cc.FORM_PERSISTENT)
    dec = _times(cands, "decompress_ms", cc.FORM_PERSISTENT)
    derived = -(-chunks // sms)
    if chunks <= sms:
        assert comp[1, 0, 0] == comp[2, 0, 0]
        assert best["form"] != cc.FORM_PERSISTENT or best["cmp_ctas"] == 2
        assert dec[0, 0, 1] == dec[0, 1, 1]  # a chunk alone, tables in HBM
        assert len({dec[0, 0, 0], dec[0, 1, 0], dec[0, 0, 1]}) == 3
    else:
        assert derived == 3
        assert comp[1, 0, 0] != comp[2, 0, 0]
        assert dec[0, 0, 0] == dec[0, 0, 1] == dec[0, derived, 0] == dec[0, derived, 1]
        assert dec[0, 1, 0] != dec[0, 1, 1]
        assert best["dec_pairs"] != derived
    for pairs in (2, 3, 4, 5):
        assert dec[0, pairs, 0] == dec[0, pairs, 1]
    assert best["dec_pairs"] < 2 or best["dec_tables"] == 0
    assert ctx.get_tuning() == best
