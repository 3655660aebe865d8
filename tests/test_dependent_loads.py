"""Kernels launched by programmatic dependent launch are resident while the
kernel before them may still write; the read-only path asks for data that
nobody writes during a kernel's whole life (CPU, the sources)."""

import os
import re

from leviathan_v1_b200._build import CSRC


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def test_dependent_kernels_gather_the_ring_by_ordinary_loads():
    text = _source("lev_pair.cuh")
    assert "wait_dependency()" in text
    assert "ld_ring_dependent(" in text and not re.search(r"\bld_ring\(", text)
    # of the read-only loads there, only the column / delay words remain
    assert set(re.findall(r"__ldg\(([a-z_]+)", text)) == {"cdp"}


def test_only_the_pair_kernels_are_launched_dependently():
    launcher = _source("lev_engine.cu")
    assert launcher.count("cudaLaunchAttributeProgrammaticStreamSerialization") == 1
    for name in os.listdir(CSRC):
        if name not in ("lev_pair.cuh", "lev_kernels.cuh"):
            assert "wait_dependency(" not in _source(name), name
