"""What a kernel's source has to say in a certain order, read as text."""
import glob
import os
import re

import pytest

from vx_b200.build import CSRC


def kernels():
    """(file, name, body) of every __global__ function that is defined in csrc."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"/\*.*?\*/|//[^\n]*", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"__global__ void\s+(?:__\w+__\([^)]*\)\s*)*(\w+)\([^;{]*\)\s*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            yield os.path.basename(path), m.group(1), text[m.end():at]


TENSOR_MEMORY = [k for k in kernels() if "tmem_alloc" in k[2]]


def test_the_kernels_on_tensor_memory_are_found():
    assert len(TENSOR_MEMORY) >= 8


@pytest.mark.parametrize("body", [pytest.param(k[2], id="%s:%s" % k[:2]) for k in TENSOR_MEMORY])
def test_a_kernel_has_its_tensor_memory_before_it_releases_the_next(body):
    """A successor that took its own first could wait for this kernel's end while this one
    waits, without a limit, for columns."""
    release = body.find("chain_release()")
    assert release < 0 or body.rfind("tmem_alloc") < release
