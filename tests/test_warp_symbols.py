"""CPU test of the context modelling's warp code (csrc/t1sym.cuh), a host thread per lane under
ThreadSanitizer with warp intrinsics that order memory only where CUDA says so: the oracle's
symbols for every form and band orientation, packed and with every pass on a 16-byte boundary, and
no two lanes' accesses that nothing but a shuffle separates."""
import os
import shutil
import struct
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or
                                not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                                reason="needs g++ and the CUDA headers")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("warp") / "warp_symbols")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(ROOT, "roger_b200", "csrc"), "-I", os.path.join(CUDA, "include"),
                        os.path.join(ROOT, "tests", "cpp", "warp_symbols.cpp"), "-o", out, "-pthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return out


def _block(w, h, orient):
    rng = np.random.default_rng(1000 * w + 10 * h + orient)
    b = (rng.random((h, w)) < 0.3) * rng.integers(-9, 10, (h, w))
    b[: (h + 1) // 2] = rng.integers(-3, 4, ((h + 1) // 2, w))
    return b.astype(np.int32)


@pytest.mark.parametrize("pad", [0, 1])
def test_symbols_equal_the_oracle_without_a_race(exe, pad):
    # both sides of the forms' limits, ragged stripes, a block of one sample
    blocks = [(w, h, o) for w, h in [(1, 1), (4, 4), (8, 3), (5, 7), (8, 16), (3, 31), (8, 61), (32, 32), (31, 9), (9, 33), (33, 6), (40, 13)] for o in range(4)]
    blocks += [(32, 64, 1), (64, 64, 3), (8, 64, 2), (9, 4, 1), (64, 16, 2), (33, 17, 1), (64, 32, 0), (40, 33, 1)]
    data = b"".join(struct.pack("<4i", w, h, o, pad) + _block(w, h, o).tobytes() for w, h, o in blocks)
    r = subprocess.run([exe], input=data, capture_output=True, env=dict(os.environ, TSAN_OPTIONS="exitcode=66"),
                       timeout=600)
    if b"unexpected memory mapping" in r.stderr:
        pytest.skip("ThreadSanitizer cannot start with this kernel's address layout")
    assert r.returncode == 0, (r.returncode, r.stderr[:4000].decode(errors="replace"))
    at = 0
    for w, h, o in blocks:
        n, = struct.unpack_from("<i", r.stdout, at)
        got = np.frombuffer(r.stdout, np.uint8, n, at + 4)
        at += 4 + n
        want = O.t1_encode(_block(w, h, o), o, want_symbols=True)[2]
        assert np.array_equal(got & 0x9F, want), (w, h, o)  # (bit 5: the sign's XOR bit, kept for raw passes)
    assert at == len(r.stdout)
