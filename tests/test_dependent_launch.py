"""Order of the set-up in kernels whose dependents may start early, read from the sources."""

import glob
import os
import re

from conftest import ROOT


def test_tensor_memory_is_allocated_before_dependents_may_start():
    kernels = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "flash_colsum_b200", "csrc", "*.cu*"))):
        with open(path) as f:
            text = f.read()
        for body in re.split(r"\b__global__\b", text)[1:]:
            alloc, launch = body.find("tmem_alloc("), body.find("grid_launch_dependents()")
            if alloc >= 0 and launch >= 0:
                assert alloc < launch, path
                kernels += 1
    assert kernels >= 3
