"""GPU tests of the stripe decoder (t1dec_stripe.cuh): every number of blocks per warp, block counts
on both sides of the rule that chooses it, ragged blocks of every edge size, against lossless
inputs and the oracle's decoder on cut blocks (integers, so equality)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from roger_b200 import codec as C
from roger_b200 import synth
from roger_b200._lib import lib

pytestmark = pytest.mark.gpu


def _ctx(lanes):
    ctx = C.Context(0)
    if lanes is not None:
        assert lib().j2k_ctx_set_tuning(ctx.h, 10, lanes) == 0
    return ctx


@pytest.mark.parametrize("lanes", [None, 0, 2, 3, 4, 8, 16, 32])
@pytest.mark.parametrize("w,h,levels,cb", [(1, 1, 0, 64), (3, 130, 1, 64), (65, 31, 2, 32), (129, 67, 3, 64),
                                           (400, 300, 2, 4), (640, 636, 1, 4)])
def test_lossless_round_trip(lanes, w, h, levels, cb):
    img = synth.gray(w, h, w + h)
    d, b = C.OCLEncoder(ctx=C.Context(0)).run_rgb(img, levels=levels, cbw=cb, cbh=cb).get_codeblocks()
    out = C.OCLDecoder(ctx=_ctx(lanes)).run(d, b, w, h, 1, levels=levels, cbw=cb, cbh=cb)
    assert np.array_equal(out[:, :, 0], img)


@pytest.mark.parametrize("lanes", [None, 2, 4, 8])
def test_cut_blocks_of_unlike_plane_counts(lanes):
    """Blocks that share a warp but differ in plane counts and in the pass they are cut after."""
    rng = np.random.default_rng(5)
    w, h = 512, 64
    coef = np.zeros((h, w), np.int32)
    for k in range(8):  # eight 64 x 64 blocks of one plane, amplitudes 1 .. 2^21
        coef[:, 64 * k:64 * k + 64] = rng.laplace(0, 2.0 ** (3 * k), (h, 64)).astype(np.int32)
    t = torch.from_numpy(coef).cuda()
    descs, data = C.bpc_encode(t, 0, cap_per_block=32768)
    descs = np.array(descs)
    cuts = [1, 4, 6, 8, 11, 2, 30, 200]
    data = data.cpu().numpy()
    want = np.zeros_like(coef)
    for k in range(8):
        descs["npasses"][k] = min(cuts[k], descs["npasses"][k])
        o, n = int(descs["offset"][k]), int(descs["length"][k])
        want[:, 64 * k:64 * k + 64] = O.t1_decode(data[o:o + n].tobytes(), int(descs["numbps"][k]),
                                                  int(descs["npasses"][k]), 0, 64, 64)
    got = C.bpc_decode(descs, torch.from_numpy(data).cuda(), w, h, 0, ctx=_ctx(lanes)).cpu().numpy()
    assert np.array_equal(got, want)
