"""Fixed-model decoding around the counts where its kernels change: a CTA per
chunk up to the SMs' number, then warps, then warps that take a second chunk."""
import pytest

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [1, 148, 149, 1185, 4736, 4737, 6000])
@pytest.mark.parametrize("kind", ["text", "random"])
def test_many_chunks(gpu_ctx, oracle_mod, chunks, kind):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT)
    pre, cs = 3000, 37
    data = (W.text(pre, 5).tobytes() + W.make(kind, chunks * cs - 5, chunks).tobytes())
    blob = oracle_mod.compress(data, cs, 128, pre, 100, fixed=True)
    assert gpu_ctx.decompress(blob) == data
