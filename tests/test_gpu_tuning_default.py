"""GPU tests of the way back from tuning: the rules that choose the tier-1 schedules of a new context
can be set again, the autotuners consider the new context's schedule, and what they keep and
report is a schedule that there is."""
import os
import re

import numpy as np
import pytest

from roger_b200 import codec as C
from roger_b200 import synth
from roger_b200._lib import lib
from roger_b200.batch import BatchEncoder

pytestmark = pytest.mark.gpu
MQ_LANES, T1D_LANES, GET_MQ_LANES = 1, 10, 6


def _images():
    descs = [dict(w=40 + 9 * i, h=70, ncomp=1 + 2 * (i % 2), kernel=53, levels=2, cb=32) for i in range(6)]
    return descs, [synth.gray(d["w"], d["h"], i) if d["ncomp"] == 1 else synth.rgb(d["w"], d["h"], (i, 1, 2, 3))
                   for i, d in enumerate(descs)]


def test_the_rules_can_be_set_again():
    descs, images = _images()
    be = BatchEncoder(descs)
    new = be.get_option(GET_MQ_LANES)
    want = be.encode(images).results(pinned=False)
    want = [(np.array(d), np.array(b)) for d, b in want]
    for lanes in (8, 32, new):
        assert lib().j2k_ctx_set_tuning(be.ctx.h, MQ_LANES, lanes) == 0
        assert be.get_option(GET_MQ_LANES) == lanes
        for (d, b), (wd, wb) in zip(be.encode(images).results(pinned=False), want):
            assert np.array_equal(d, wd) and np.array_equal(b, wb)
    for lanes in (4, -1):
        assert lib().j2k_ctx_set_tuning(be.ctx.h, T1D_LANES, lanes) == 0
    for key, value in ((MQ_LANES, 5), (MQ_LANES, -1), (T1D_LANES, 1), (T1D_LANES, -2)):
        assert lib().j2k_ctx_set_tuning(be.ctx.h, key, value) != 0


def test_tuned_small_batches_are_the_same_bytes_and_say_what_runs():
    descs, images = _images()
    be = BatchEncoder(descs)
    want = [(np.array(d), np.array(b)) for d, b in be.encode(images).results(pinned=False)]
    rep = be.autotune(reps=1)
    for (d, b), (wd, wb) in zip(be.encode(images).results(pinned=False), want):
        assert np.array_equal(d, wd) and np.array_equal(b, wb)
    lanes = be.get_option(GET_MQ_LANES)
    assert lanes in (0, 8, 16, 32)
    assert rep["mq"].startswith(f"{lanes} blocks per warp pair" if lanes else "1 to 32, by their number,")


def test_tuned_small_images_are_the_same_bytes():
    img = synth.gray(200, 130, 3)
    enc = C.OCLEncoder(ctx=C.Context(0))
    want = [np.array(v) for v in enc.run_rgb(img, levels=3, cbw=32, cbh=32).get_codeblocks()]
    assert enc.autotune(reps=1)["blocks_per_warp"] in (8, 16, 32)
    got = enc.run_rgb(img, levels=3, cbw=32, cbh=32).get_codeblocks()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_a_new_context_s_schedule_is_among_the_candidates():
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(C.__file__))), "roger_b200", "csrc")
    for name, row in (("codec.cu", r"\{1, 0, 0, 0\}"), ("batch.cu", r"\{0, 1\}")):
        assert re.search(r"const int cand\[\w+\]\[\d\] = \{[^;]*" + row, open(os.path.join(csrc, name)).read()), name
