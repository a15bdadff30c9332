"""CPU test of the MQ encoder the device kernels run (csrc/mq_enc.cuh, host-callable): byte for
byte the codewords of the flowcharts of T.800 Annex C.2."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "bin", "nvcc")) or shutil.which("g++") is None,
                    reason="needs nvcc and g++")
def test_mq_encoder_matches_the_flowcharts(tmp_path):
    exe = str(tmp_path / "mq_encode")
    for cmd in ([os.path.join(CUDA, "bin", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                 "-I", os.path.join(ROOT, "roger_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "mq_encode.cu"),
                 "-o", exe], [exe, "100000"]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, (r.stdout[-1000:], r.stderr[-3000:])
    assert int(r.stdout.split()[1]) == 100000
