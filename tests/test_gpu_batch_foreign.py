"""GPU tests of the images that the batched encoder's upload copies one by one, not by its gather kernel:
managed memory, the same code-blocks, and a few images alone, as fast as a copy."""
import ctypes

import numpy as np
import pytest
import torch

from roger_b200 import synth
from roger_b200._lib import lib
from roger_b200.batch import BatchEncoder

pytestmark = pytest.mark.gpu


def test_managed_images_beside_device_images():
    descs = [dict(w=61 + 10 * i, h=45, ncomp=1, kernel=53, levels=2, cb=32) for i in range(5)]
    host = [synth.gray(d["w"], d["h"], i) for i, d in enumerate(descs)]
    be = BatchEncoder(descs)
    want = [(np.array(d), np.array(b)) for d, b in be.encode(host).results(pinned=False)]
    be.encode([np.zeros_like(im) for im in host])
    keep, ptrs, managed = [], (ctypes.c_void_p * 5)(), ctypes.c_void_p()
    rt = lib()  # (the runtime is one of the library's own)
    assert rt.cudaMallocManaged(ctypes.byref(managed), ctypes.c_size_t(1 << 16), ctypes.c_uint(1)) == 0
    try:
        at = managed.value
        for i, im in enumerate(host):
            if i % 2:
                ctypes.memmove(at, im.ctypes.data, im.size)
                ptrs[i] = at
                at += im.size
            else:
                keep.append(torch.from_numpy(im).cuda())
                ptrs[i] = keep[-1].data_ptr()
        torch.cuda.synchronize()
        assert lib().j2k_batch_upload(be.h, ptrs, 1) == 0
        got = be.encode(None).results(pinned=False)
        for (d, b), (wd, wb) in zip(got, want):
            assert np.array_equal(d, wd) and np.array_equal(b, wb)
    finally:
        torch.cuda.synchronize()
        assert rt.cudaFree(managed) == 0


def _upload_time(images):
    be = BatchEncoder([dict(w=im.shape[1], h=im.shape[0], ncomp=3, kernel=53, levels=1, cb=64) for im in images])
    best = 1e30
    for _ in range(20):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        be.upload(images)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_one_image_off_a_16_byte_boundary_uploads_like_a_copy():
    """4096 x 4096 colour at 8 mod 16: 41 us by the gather kernel, 24 by a copy."""
    n = 3 * 4096 * 4096
    pool = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
    t = [_upload_time([pool[at:at + n].view(4096, 4096, 3)]) for at in (0, 8)]
    assert t[1] < 1.35 * t[0], t


@pytest.mark.parametrize("n", [1, 3, 4])
def test_few_device_images(n):
    descs = [dict(w=33 + i, h=40, ncomp=1, kernel=53, levels=1, cb=32) for i in range(n)]
    host = [synth.gray(d["w"], d["h"], i) for i, d in enumerate(descs)]
    a = [(np.array(d), np.array(b)) for d, b in BatchEncoder(descs).encode(host).results(pinned=False)]
    b = BatchEncoder(descs).encode([torch.from_numpy(im).cuda() for im in host]).results(pinned=False)
    for (da, ba), (db, bb) in zip(a, b):
        assert np.array_equal(da, db) and np.array_equal(ba, bb)
