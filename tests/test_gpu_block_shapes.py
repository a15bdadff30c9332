"""GPU tests of code-blocks of every shape: the forms the tier-1 kernels choose by a block's width and
height, against the oracle and lossless inputs (bytes and integers, so equality), and that no
shape costs a multiple of what another one of as many samples does."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from roger_b200 import codec as C
from roger_b200 import synth
from roger_b200._lib import lib

from test_gpu_t1_symbols import _contents

pytestmark = pytest.mark.gpu


def _time(fn):
    """Least of 7 runs, in ms on the device."""
    fn()
    best = 1e30
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("w,h", [(33, 17), (64, 32), (64, 16), (40, 33), (8, 4), (8, 5), (4, 4), (9, 4), (8, 64), (7, 9)])
def test_encoded_blocks_equal_oracle(w, h):
    for name, blk in _contents(w, h).items():
        for levels in (0, 1):
            coef = np.ascontiguousarray(np.tile(blk, (1 << levels, 1 << levels)))
            descs, data = C.bpc_encode(torch.from_numpy(coef).cuda(), levels, cap_per_block=32768)
            data = data.cpu().numpy()
            for d in descs:
                want, info = O.t1_encode(blk, int(d["orient"]))
                assert (d["numbps"], d["npasses"]) == (info["numbps"], info["npasses"]), (name, d)
                assert data[d["offset"]:d["offset"] + d["length"]].tobytes() == want, (name, int(d["orient"]))


@pytest.fixture(scope="module")
def picture():
    return torch.from_numpy(synth.rgb(1024, 1024, (1, 2, 3, 4))).cuda()


# with one lane of a warp in 16 or 32 at work: 1.8 and 2.1; with the forms by shape 1.0 and 1.3 (and 8 x 8
# blocks, since then faster themselves, 1.5)
@pytest.mark.parametrize("shape,other,most", [((64, 4), (16, 16), 1.4), ((4, 4), (8, 8), 1.7)])
def test_no_shape_encodes_much_slower(picture, shape, other, most):
    enc = C.OCLEncoder(ctx=C.Context(0))
    t = [_time(lambda: enc.run_rgb(picture, levels=5, cbw=cw, cbh=ch)) for cw, ch in (shape, other)]
    assert t[0] < most * t[1], t


def _decoding(img, cbw, cbh, lanes=None, lossy=False):
    """A call that decodes img coded with blocks of cbw x cbh, with the tuned number of blocks per warp."""
    h, w, n = img.shape
    enc = C.OCLEncoder(ctx=C.Context(0), lossy=lossy).run_rgb(img, levels=5, cbw=cbw, cbh=cbh)
    d, b = [np.array(v) for v in enc.get_codeblocks()]
    ctx = C.Context(0)
    if lanes is not None:
        assert lib().j2k_ctx_set_tuning(ctx.h, 10, lanes) == 0
    dec, out = C.OCLDecoder(ctx=ctx, lossy=lossy), torch.empty((h, w, n), dtype=torch.uint8, pin_memory=True).numpy()
    return lambda: dec.run(d, b, w, h, n, levels=5, cbw=cbw, cbh=cbh, out=out)


# with the work counted in blocks of 64 x 64: 2.0 and 1.5; in blocks of the largest one's size 1.0
@pytest.mark.parametrize("size,cb", [(1024, 16), (2048, 32)])
def test_blocks_per_warp_fit_small_blocks(size, cb):
    img = torch.from_numpy(synth.rgb(size, size, (1, 2, 3, 4))).cuda()
    t = [_time(_decoding(img, cb, cb, lanes)) for lanes in (None, 2, 4)]
    assert t[0] < 1.2 * min(t[1:]), t


# 49152 blocks either way: 2.3 with the form for 64 columns, 0.8 with that for 8
def test_narrow_blocks_decode_as_fast_as_wide_ones():
    img = torch.from_numpy(synth.rgb(2048, 2048, (1, 2, 3, 4))).cuda()
    t = [_time(_decoding(img, cw, ch)) for cw, ch in ((4, 64), (64, 4))]
    assert t[0] < 1.15 * t[1], t


@pytest.mark.parametrize("lanes", [None, 0, 2, 4, 8, 16])
@pytest.mark.parametrize("w,h,cbw,cbh", [(1, 1, 4, 4), (70, 50, 4, 64), (133, 65, 8, 8), (260, 131, 8, 64), (400, 300, 8, 4)])
def test_narrow_blocks_round_trip(lanes, w, h, cbw, cbh):
    img = torch.from_numpy(synth.rgb(w, h, (w, h, 3, 4))).cuda()
    assert np.array_equal(_decoding(img, cbw, cbh, lanes)(), img.cpu().numpy())


# the numbers of blocks on both sides of every line of the rule (148 SMs: 2368, 7104, 14208, 37888)
@pytest.mark.parametrize("blocks", [2300, 2400, 7000, 7200, 14100, 14300, 37800, 38000])
def test_narrow_blocks_of_every_count(blocks):
    w, h = 4 * 100, 4 * (blocks // 100)
    img = synth.gray(w, h, blocks)
    d, b = C.OCLEncoder(ctx=C.Context(0)).run_rgb(img, levels=0, cbw=4, cbh=4).get_codeblocks()
    assert len(d) == blocks
    out = C.OCLDecoder(ctx=C.Context(0)).run(d, b, w, h, 1, levels=0, cbw=4, cbh=4)
    assert np.array_equal(out[:, :, 0], img)


@pytest.mark.parametrize("lanes", [None, 2, 16])
@pytest.mark.parametrize("style", [1, 6, 7])
def test_narrow_blocks_with_styles(lanes, style):
    img = synth.rgb(150, 101, (5, 6, 7, 8))
    enc = C.OCLEncoder(ctx=C.Context(0)).run_rgb(img, levels=3, cbw=8, cbh=64, cblk_style=style)
    d, b = enc.get_codeblocks()
    ctx = C.Context(0)
    if lanes is not None:
        assert lib().j2k_ctx_set_tuning(ctx.h, 10, lanes) == 0
    out = C.OCLDecoder(ctx=ctx).run(d, b, 150, 101, 3, levels=3, cbw=8, cbh=64, cblk_style=style,
                                    pass_ends=enc.get_pass_ends())
    assert np.array_equal(out, img)


@pytest.mark.parametrize("lanes", [None, 4, 16])
def test_narrow_blocks_cut_after_any_pass(lanes):
    """Blocks that share a warp but differ in plane counts and in the pass they are cut after."""
    rng = np.random.default_rng(5)
    coef = np.concatenate([rng.laplace(0, 2.0 ** k, (64, 8)).astype(np.int32) for k in range(22)], 1)
    descs, data = C.bpc_encode(torch.from_numpy(coef).cuda(), 0, cbw=8, cbh=64, cap_per_block=8192)
    descs, data, want = np.array(descs), data.cpu().numpy(), np.zeros_like(coef)
    for k in range(22):
        descs["npasses"][k] = min(1 + 3 * int(rng.integers(0, 20)) + k % 3, descs["npasses"][k])
        o, n = int(descs["offset"][k]), int(descs["length"][k])
        want[:, 8 * k:8 * k + 8] = O.t1_decode(data[o:o + n].tobytes(), int(descs["numbps"][k]),
                                               int(descs["npasses"][k]), 0, 8, 64)
    ctx = C.Context(0)
    if lanes is not None:
        assert lib().j2k_ctx_set_tuning(ctx.h, 10, lanes) == 0
    got = C.bpc_decode(descs, torch.from_numpy(data).cuda(), 176, 64, 0, cbw=8, cbh=64, ctx=ctx).cpu().numpy()
    assert np.array_equal(got, want)


def test_one_large_block_among_many_small_ones():
    """The blocks per warp follow the many."""
    imgs = [(synth.gray(512, 512, k), 16) for k in range(30)] + [(synth.gray(64, 64, 99), 64)]
    streams = [C.OCLEncoder(ctx=C.Context(0)).run_rgb(im, levels=1, cbw=cb, cbh=cb).codestream() for im, cb in imgs]
    t = []
    for lanes in (None, 4):
        ctx = C.Context(0)
        if lanes is not None:
            assert lib().j2k_ctx_set_tuning(ctx.h, 10, lanes) == 0
        dec = C.OCLDecoder(ctx=ctx)
        t.append(_time(lambda: C.decode_codestreams(streams, decoder=dec)))
        for (im, _), out in zip(imgs, C.decode_codestreams(streams, decoder=dec)):
            assert np.array_equal(np.array(out).reshape(im.shape), im)
    assert t[0] < 1.2 * t[1], t
