"""GPU test of the batched encoder's upload from memory that is not the device's own (managed memory):
copied image by image, beside images that the gather kernel takes, the same code-blocks."""
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
