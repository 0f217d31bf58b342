"""A source rule of the programmatic launches, checked without a GPU.

A read through a __restrict__ pointer is not held back by pdl_wait() (see
common.cuh), so every kernel that waits and has such a parameter forms its
addresses from a value that passed after_wait() below the wait.  And a kernel
that is launched programmatically waits at all."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "bootcmatchg_b200", "csrc")


def closing(s, i, pair):
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == pair[0]) - (s[k] == pair[1])
        if depth == 0:
            return k
    raise ValueError("unbalanced")


def kernels(path):
    """(name, parameter list, body) of every __global__ function."""
    s = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__global__", s):
        name = re.compile(r"\b(k_\w+)\s*\(").search(s, m.end())
        p1 = closing(s, name.end() - 1, "()")
        b0 = s.index("{", p1)
        yield name.group(1), s[name.end():p1], s[b0:closing(s, b0, "{}")]


FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_reads_of_waiting_kernels_start_below_the_wait(path):
    for name, params, body in kernels(path):
        if "pdl_wait()" in body and "__restrict__" in params:
            after = body[body.rindex("pdl_wait()"):]
            assert "after_wait(" in after, name


def test_programmatically_launched_kernels_wait():
    waits = {n: "pdl_wait()" in b for f in FILES for n, _, b in kernels(f)}
    launched = set()
    for f in FILES:
        launched |= set(re.findall(r"launch_pdl\(\s*(k_\w+)", open(f).read()))
    assert len(launched) > 30
    assert not [k for k in launched if not waits[k]]
