"""The fixed-model coder with a warp per chunk: chunk lengths around the 32 bytes
it takes at a time and the 512 it writes at a time, data the model does not
expect, and the counts around where chunks share warps."""
import pytest

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(ctx, oracle, data, cs, pre):
    ctx.set_tuning(form=cc.FORM_PERSISTENT)
    want = oracle.compress(data, cs, 128, pre, 100, fixed=True)
    assert ctx.compress(data, cs, 128, pre, 100, fixed=True) == want
    assert ctx.decompress(want) == data


@pytest.mark.parametrize("cs", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 511, 513, 4097])
@pytest.mark.parametrize("kind", ["text", "random"])
def test_lengths(gpu_ctx, oracle_mod, cs, kind):
    data = W.text(2000, 9).tobytes() + W.make(kind, 5 * cs + cs // 2, cs).tobytes()
    _check(gpu_ctx, oracle_mod, data, cs, 2000)


@pytest.mark.parametrize("chunks", [591, 592, 593])
def test_counts(gpu_ctx, oracle_mod, chunks):
    data = W.text(2000, 9).tobytes() + W.make("text", 43 * chunks - 20, chunks).tobytes()
    _check(gpu_ctx, oracle_mod, data, 43, 2000)


@pytest.mark.parametrize("n", [32768, 70001])
def test_unexpected(gpu_ctx, oracle_mod, n):
    _check(gpu_ctx, oracle_mod, bytes(16384) + b"\xff" * n, 32768, 16384)
