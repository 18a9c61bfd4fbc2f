"""What a kernel owes the launch in front of it when its set-up runs beside that one's end
(launch_after, host_common.h), read from the sources: running a kernel that breaks it would be a race."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ptx.jl_b200", "csrc")


def code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


FILES = [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu") and "launch_after(" in code(f)]


def test_files():
    assert len(FILES) == 5


@pytest.mark.parametrize("name", FILES + ["gemm_epilogue.cuh", "sm100_prims.cuh"])
def test_no_read_only_loads(name):
    """The read-only path wants memory that nothing writes while the kernel runs, and it runs from
    before the end of the kernel in front: no ld.global.nc, and nothing the compiler makes one of."""
    text = code(name)
    assert "__ldg(" not in text and not re.search(r"ld\.global[.\w]*\.nc\b", text)
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", text)
