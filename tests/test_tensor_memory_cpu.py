"""Kernels that take tensor memory let their successor start only once they have it (tcgen05.cuh says why): read off the sources."""
import os
import re

from denograd_b200 import build as B


def test_successors_start_behind_the_allocation():
    seen = 0
    for name in sorted(os.listdir(B.CSRC)):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(B.CSRC, name)).read())
        for body in re.split(r"__global__|\ntemplate <", src):
            if "tcgen05.alloc" not in body:
                continue
            seen += 1
            begin = body.index("tcgen05.alloc")
            assert "pdl_launch()" in body[begin:] and "pdl_launch()" not in body[:begin], name
            # behind a barrier of all warps, one of which allocates
            assert "__syncthreads()" in body[begin:body.index("pdl_launch()")], name
    assert seen == 4
