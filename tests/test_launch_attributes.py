"""What a launcher sets once is set once on each device: a kernel's share of shared memory belongs to the device that was current when it was asked for."""
import os
import re

import pytest

from velomind_b200.kernels import library

FILES = sorted(f for f in os.listdir(library.CSRC) if f.endswith((".cu", ".cuh")))


@pytest.mark.parametrize("name", FILES)
def test_no_launcher_remembers_an_attribute_for_the_process(name):
    """An attribute set behind a plain static is missing on a second device, whose launches are then refused.  Launchers ask through vm_allow_smem (done once on
    each device, tests/cpp/host_tests.cpp) or at every launch."""
    lines = open(os.path.join(library.CSRC, name)).read().splitlines()
    for i, line in enumerate(lines):
        if "cudaFuncSetAttribute" in line and name != "common.cuh":
            before = "\n".join(lines[max(0, i - 5):i + 1])
            assert not re.search(r"static\s+(bool|int|size_t)\b", before), f"{name}:{i + 1}"
