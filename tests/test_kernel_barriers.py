"""CPU checks of the kernels' source for barriers that CUDA leaves undefined or that are missing."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "roger_b200", "csrc")


def _code():
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        yield os.path.basename(f), re.sub(r"//[^\n]*", "", open(f).read())


def _end_of_block(src, at):
    """Position after the brace that closes the block opened at src[at]."""
    depth = 0
    for i in range(at, len(src)):
        depth += (src[i] == "{") - (src[i] == "}")
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced braces")


def test_no_block_barrier_where_the_warps_part():
    """__syncthreads is defined only where all threads of the block come to the same one: warps that
    take different roles meet at numbered barriers instead."""
    roles = 0
    for name, src in _code():
        for m in re.finditer(r"\bif \(threadIdx\.x < 32\) \{", src):
            end = _end_of_block(src, m.end() - 1)
            arm = src[m.end():end]
            roles += 1
            assert "__syncthreads" not in arm, name
            if re.search(r"return;\s*\}$", arm):  # the other warps' role is the rest of the kernel
                rest = src[end:src.index("\n}\n", end)]
                assert "__syncthreads" not in rest, name
    assert roles > 0


def test_strips_that_tensor_copies_refill_are_fenced():
    """A thread that has written shared memory which a tensor copy then overwrites puts a proxy fence
    before the barrier after which the copy is issued: a barrier alone does not order the two."""
    loops = 0
    for name, src in _code():
        for m in re.finditer(r"cp\.async\.bulk\.tensor", src):
            start = src.rindex("__global__", 0, m.start())
            body = src[start:_end_of_block(src, src.index("{", src.index(")", start)))]
            assert re.search(r"fence_proxy_async\(\);\s*__syncthreads\(\);\s*\}\s*\}$", body), name
            loops += 1
    assert loops > 0
