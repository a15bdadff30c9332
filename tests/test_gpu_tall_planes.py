"""GPU test of planes so high that the strips of a level would be more rows than a grid has: they take
the tile kernel (integers, so equality)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from roger_b200 import codec as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [16 * 65535, 16 * 65535 + 1])
def test_tall_planes_of_odd_width_forward(h):
    x = np.random.default_rng(h).integers(-128, 128, (h, 9)).astype(np.int32)
    y = C.dwt_forward(torch.from_numpy(x).cuda(), 2).cpu().numpy()
    assert np.array_equal(y, O.dwt53_fwd(x, 2))
