"""Every unit length of the pipelined kernels, at chunk lengths around whole
units: the slot numbers a unit's bits share (few distinct slots in runs, nearly
all distinct in random bytes, repeats across units in text), the last unit's
missing bits, and the link to the unit before.  Containers equal the oracle's
byte for byte and decode back."""
import pytest

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [32, 64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("kind", ["text", "runs", "random", "walk"])
def test_unit_lengths(gpu_ctx, oracle_mod, unit, kind):
    ub = unit // 8
    for form in (cc.FORM_PERSISTENT, cc.FORM_PLAIN):
        gpu_ctx.set_tuning(form=form)
        for n, cs in ((ub * 40 + 1, ub * 40 + 1), (ub * 9 - 1, ub * 9 - 1), (ub, ub), (1, ub + 1), (7000, 2048)):
            data = W.make(kind, n, n + unit).tobytes()
            want = oracle_mod.compress(data, cs, unit, 0, 100)
            assert gpu_ctx.compress(data, cs, unit) == want
            assert gpu_ctx.decompress(want) == data
