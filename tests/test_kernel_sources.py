"""What the kernels' sources must keep to where no run shows that they do."""
import glob
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "csrc", "kernels")


def _issuing_kernels():
    """(file, name, body) of every kernel in which one elected thread of a warp issues copies or MMAs."""
    for path in sorted(glob.glob(os.path.join(KERNELS, "*.cu"))):
        with open(path) as f:
            parts = f.read().split("__global__")[1:]
        for body in parts:
            if "elect_one()" in body:
                name = re.search(r"\b(\w+_kernel)\b", body).group(1)
                yield pytest.param(body, id=os.path.basename(path) + ":" + name)


@pytest.mark.parametrize("body", list(_issuing_kernels()))
def test_issuing_warps_are_whole_at_aligned_barriers(body):
    """`bar.sync` and `barrier.cluster` of the inline PTX are aligned: all lanes of a warp execute them together.  The lanes that were
    not elected skip the issuing loop, so a warp has to come together again before the first barrier that it shares with the others."""
    tail = body[body.rindex("elect_one()"):]
    m = re.search(r"cluster_arrive\(\)|named_bar_sync\(\d+, k\w*Threads\)", tail)
    if m is None:
        return
    before = tail[:m.start()].splitlines()[-6:]
    assert any("__syncwarp();" in line or "__syncthreads();" in line for line in before), "\n".join(before)
