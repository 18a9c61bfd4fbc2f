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


def kernels(text):
    """(name, body) of the file's kernels."""
    for part in text.split("__global__ void")[1:]:
        name = re.search(r"\w+_kernel(?=\()", part)
        start = part.index(") {\n", name.end()) + 2
        yield name.group(), part[start:part.index("\n}\n", start)]


def enclosing(body, at):
    """The text of the block that holds position `at`, from its opening brace on up to there."""
    depth, i = 0, at
    while True:
        i -= 1
        if body[i] == "}":
            depth += 1
        elif body[i] == "{":
            if depth == 0:
                return body[i:at]
            depth -= 1


@pytest.mark.parametrize("name", FILES)
def test_nothing_is_written_and_nobody_leaves_ahead_of_the_wait(name):
    """The launch behind waits for this one's end and no more: were all of a launch's threads to leave
    without a wait for the kernel in front, it would run beside that one."""
    found = list(kernels(code(name)))
    assert found
    for kernel, body in found:
        assert "grid_wait();" in body, kernel
        for m in re.finditer(r"\batomicCAS\(|\breturn;", body):
            assert "grid_wait();" in enclosing(body, m.start()), (kernel, body[m.start() - 80:m.end()])
