"""GPU test of the bit-sliced context modelling (t1sym.cuh) and the warp-pair MQ coder behind it: each
form a block's shape selects, at its edges, on contents from empty to more symbols than one staging
round holds, against the oracle's coder (bytes, so equality)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from roger_b200 import codec as C

pytestmark = pytest.mark.gpu


def _contents(w, h):
    rng = np.random.default_rng(100 * w + h)
    point = np.zeros((h, w), np.int32)
    point[h - 1, w - 1] = -5
    rows = np.zeros((h, w), np.int32)
    rows[::4] = (1 << 12) - 1
    return {
        "empty": np.zeros((h, w), np.int32),
        "point": point,
        "rows": rows,
        "sparse": (rng.random((h, w)) < 0.02).astype(np.int32) * rng.integers(-300, 300, (h, w)).astype(np.int32),
        "noise": rng.integers(-(1 << 20), 1 << 20, (h, w)).astype(np.int32),
        "bits": rng.integers(-1, 2, (h, w)).astype(np.int32),
    }


@pytest.mark.parametrize("w,h", [(64, 64), (33, 64), (63, 61), (32, 64), (31, 33), (32, 32), (5, 32), (1, 1), (64, 1),
                                 (1, 64), (17, 3), (40, 5)])
@pytest.mark.parametrize("levels", [0, 1])
def test_blocks_of_every_shape_equal_oracle(w, h, levels):
    for name, blk in _contents(w, h).items():
        # levels 1: the same block as HL, LH and HH (and as LL), whose context tables differ
        coef = np.tile(blk, (1 << levels, 1 << levels))
        descs, data = C.bpc_encode(torch.from_numpy(np.ascontiguousarray(coef)).cuda(), levels, cap_per_block=32768)
        data = data.cpu().numpy()
        assert len(descs) == 4 ** levels
        for d in descs:
            want, info = O.t1_encode(blk, int(d["orient"]))
            assert (d["numbps"], d["npasses"]) == (info["numbps"], info["npasses"]), (name, d)
            assert data[d["offset"]:d["offset"] + d["length"]].tobytes() == want, (name, int(d["orient"]))
