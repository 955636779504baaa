"""Containers in device memory with many batches: payloads shorter and longer
than the pieces their framing is fetched in."""
import numpy as np
import pytest
import torch

import cucm_b200 as cc
from cucm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cs,batch,kind", [(60000, 100, 1, "text"), (60000, 100, 3, "random"),
                                             (400000, 5000, 1, "random"), (900000, 34000, 1, "random"),
                                             (900000, 50000, 1, "random"), (900000, 10000, 2, "text")])
@pytest.mark.parametrize("fmt", [cc.FORMAT_32, cc.FORMAT_64])
def test_many_batches(gpu_ctx, n, cs, batch, kind, fmt):
    gpu_ctx.set_tuning(form=cc.FORM_PERSISTENT)
    pre = 500
    data = np.concatenate([W.text(pre, 1), W.make(kind, n, n + cs)])
    blob = gpu_ctx.compress(data, cs, 64, pre, batch, fmt, fixed=True)
    d_in = torch.from_numpy(np.frombuffer(blob, dtype=np.uint8).copy()).cuda()
    d_out = torch.zeros(data.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert gpu_ctx.decompress_dev(d_in.data_ptr(), len(blob), d_out.data_ptr(), data.size) == data.size
    assert d_out.cpu().numpy().tobytes() == data.tobytes()
    for cut in (len(blob) // 3, len(blob) - 1):
        with pytest.raises(cc.CucmError) as e:
            gpu_ctx.decompress_dev(d_in.data_ptr(), cut, d_out.data_ptr(), data.size)
        assert e.value.status == cc.EFORMAT
