"""Containers in device memory whose framing does not lie in their first
bytes: a long prelearn block (coded or raw), batch tables longer than 4 KiB,
many batches, the 64-bit container, and truncations in each."""
import numpy as np
import pytest
import torch

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = [(30000, 16, 0, 3000, cc.FORMAT_32), (30000, 16, 0, 7, cc.FORMAT_32), (40000, 1000, 9000, 5, cc.FORMAT_32),
         (30000, 16, 0, 1100, cc.FORMAT_64), (40000, 1000, 9000, 100, cc.FORMAT_64), (100, 64, 0, 1, cc.FORMAT_32)]


@pytest.mark.parametrize("n,cs,pre,batch,fmt", CASES)
@pytest.mark.parametrize("kind", ["text", "random"])  # random: the prelearn block stays raw
def test_device_container(gpu_ctx, n, cs, pre, batch, fmt, kind):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT)
    data = W.make(kind, n, n + cs)
    blob = gpu_ctx.compress(data, cs, 64, pre, batch, fmt)
    d_in = torch.from_numpy(np.frombuffer(blob, dtype=np.uint8).copy()).cuda()
    d_out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert gpu_ctx.decompress_dev(d_in.data_ptr(), len(blob), d_out.data_ptr(), n) == n
    assert d_out.cpu().numpy().tobytes() == data.tobytes()
    for cut in (10, len(blob) // 2, len(blob) - 1):
        with pytest.raises(cc.CucmError) as a:
            gpu_ctx.decompress(blob[:cut])
        with pytest.raises(cc.CucmError) as b:
            gpu_ctx.decompress_dev(d_in.data_ptr(), cut, d_out.data_ptr(), n)
        assert a.value.status == b.value.status == cc.EFORMAT
