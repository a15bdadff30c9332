"""GPU test of the forward level kernel on planes of any pitch: the default form loads single
samples, so odd widths (odd pitches, unaligned rows and planes) take it too.  Integers and
separately rounded FP32 operations in the oracle's order, so equality."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from roger_b200 import codec as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h,levels", [(1, 9, 2, 1), (1, 247, 16, 2), (1, 249, 17, 3), (3, 251, 33, 4),
                                          (2, 497, 31, 5), (1, 1025, 255, 6), (3, 8, 7, 2)])
def test_odd_planes_forward_and_back(n, w, h, levels):
    rng = np.random.default_rng(w * h)
    x = rng.integers(-128, 128, (n, h, w)).astype(np.int32)
    for dtype, fwd in ((np.int32, O.dwt53_fwd), (np.float32, O.dwt97_fwd)):
        xi = x.astype(dtype)
        t = torch.from_numpy(xi).cuda()
        y = C.dwt_forward(t, levels)
        for k in range(n):
            assert np.array_equal(y[k].cpu().numpy(), fwd(xi[k], levels))
        # a view whose first sample is not 16-byte aligned
        pad = torch.zeros((n, h, w + 3), dtype=t.dtype, device="cuda")
        pad[:, :, 1:w + 1] = t
        assert torch.equal(C.dwt_forward(pad[:, :, 1:w + 1], levels), y)
        back = C.dwt_inverse(y, levels)
        if dtype is np.int32:
            assert torch.equal(back, t)
