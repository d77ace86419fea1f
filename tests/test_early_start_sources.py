"""Kernels that may start under the tail of the launch before them (programmatic launches) wait before they touch what earlier launches
wrote.  `__restrict__` promises the compiler that nobody else writes the data while the kernel lives, which is not so before the
wait, and loads through such pointers were moved ahead of it.  A race is not something a test can wait for: the sources are read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kfold_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("kernel", ["adaln_vec_kernel", "adaln_rows_kernel"])
def test_adaln_makes_no_promise_about_its_inputs(kernel):
    params = re.search(r"__global__[^;{]*?\b%s\s*\((.*?)\)\s*\{" % kernel, source("layernorm.cu"), flags=re.S).group(1)
    assert "gv" in params and "__restrict__" not in params
