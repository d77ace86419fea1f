"""Kernels that may start under the tail of the launch before them (programmatic launches) wait before they touch what earlier launches
wrote.  `__restrict__`, `__ldg` and `ld.global.nc` promise the compiler that nobody else writes the data while the kernel lives, which is
not so before the wait, and it moved loads ahead of it.  A race is not something a test can wait for: the sources are read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kfold_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


NAMES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
EARLY = [n for n in NAMES if "grid_dependency_" in source(n)]


@pytest.mark.parametrize("name", EARLY)
def test_no_promise_about_data_of_the_launch_before(name):
    assert not re.findall(r"__restrict__|__ldg\b|ld\.global\.nc", source(name))


@pytest.mark.parametrize("name", [n for n in NAMES if "__global__" in source(n)])
def test_kernels_that_do_not_wait_are_launched_plainly(name):
    """Every kernel of a file waits and is launched by launch_kernel, or none does either."""
    text = source(name)
    kernels = re.findall(r"__global__[^;{]*?\b(\w+)\s*\((?:[^(){}]|\([^()]*\))*\)\s*\{", text)
    bodies = re.split(r"__global__", text)[1:]
    assert len(kernels) == len(bodies)
    if name in EARLY:
        for kernel, body in zip(kernels, bodies):
            assert "grid_dependency_" in body, kernel
    else:
        assert "launch_kernel" not in text
