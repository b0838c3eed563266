"""Rules of the CUDA sources that no run shows when they are broken."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pde_module_b200", "csrc")


def _kernels():
    """(name, signature, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in text.split("__global__")[1:]:
            signature, body = part.split("{", 1)
            yield re.search(r"(\w+_kernel)\s*\(", signature).group(1), signature, body


def test_no_read_only_pointers_under_an_early_launch():
    """A kernel that waits for its predecessor may be resident while that one writes: no
    pointer of it may promise constant data."""
    early = []
    for name, signature, body in _kernels():
        if "pdl_wait()" in body:
            early.append(name)
            assert not re.search(r"const float\s*\*\s*__restrict__", signature), name
            assert "__ldg" not in body, name
    assert len(early) >= 10
