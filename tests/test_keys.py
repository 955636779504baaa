"""The 8 bits of a byte never share a table slot: for one context the hash is
one-to-one in the partial byte (the compressor's walker and the decoder's
updater take a byte's or a nibble's bits together on the strength of it)."""
import numpy as np
import pytest


@pytest.mark.parametrize("seed", range(4))
def test_partial_bytes_never_collide(seed):
    rng = np.random.default_rng(seed)
    m = np.uint32((1 << 25) - 1)
    h0 = np.arange(1, 256, dtype=np.uint32)
    for _ in range(200):
        acc = (np.uint32(2166136261) ^ h0) * np.uint32(16777619)
        hist = rng.integers(0, 256, size=7).astype(np.uint32)
        if seed == 3:
            hist = rng.choice(np.array([0, 255], dtype=np.uint32), size=7)
        for c in hist:
            acc = (acc ^ c) * np.uint32(16777619)
            assert len(np.unique(acc & m)) == 255
