"""GPU test of the batched encoder's image gather: device images of any size and alignment (more than
one launch holds), the same code-blocks as from host memory."""
import numpy as np
import pytest
import torch

from roger_b200.batch import BatchEncoder

pytestmark = pytest.mark.gpu


def test_device_images_of_any_size_and_alignment():
    rng = np.random.default_rng(3)
    descs, host, dev = [], [], []
    pool = torch.zeros(1 << 21, dtype=torch.uint8, device="cuda")
    at = 0
    for i in range(131):  # two launches of the gather
        w, h, c = (300, 221, 3) if i == 7 else (int(rng.integers(1, 40)), int(rng.integers(1, 40)), 1 + 2 * (i % 2))
        im = rng.integers(0, 256, (h, w, c) if c == 3 else (h, w)).astype(np.uint8)
        descs.append(dict(w=w, h=h, ncomp=c, kernel=53, levels=1, cb=32))
        host.append(im)
        t = pool[at:at + im.size].view(im.shape)  # back to back: every alignment
        t.copy_(torch.from_numpy(im))
        dev.append(t)
        at += im.size
    a = BatchEncoder(descs).encode(host).results(pinned=False)
    b = BatchEncoder(descs).encode(dev).results(pinned=False)
    for (da, ba), (db, bb) in zip(a, b):
        assert np.array_equal(da, db) and np.array_equal(ba, bb)
