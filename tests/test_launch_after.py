"""The launch that every kernel goes through (launch_after, host_common.h), compiled on the host
against a runtime of the test's own."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("launch") / "launch_after")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ptx.jl_b200", "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "host", "launch_after.cpp"), "-o", exe], check=True)
    return subprocess.run([exe], check=True, stdout=subprocess.PIPE, text=True).stdout.splitlines()


def test_what_the_runtime_is_handed(lines):
    assert lines[:2] == ["launch 3 128 4096 7 1 after 1", "launch 8 64 0 9 1 after 1 cluster 4"]


def test_a_failed_launch_leaves_no_error_for_the_next_check(lines):
    """It is reported as the call's own result; whoever checks the runtime's last error next (the
    framework, behind a kernel of its own) does not find it there."""
    outcomes = [line.split() for line in lines if line.startswith("returned")]
    assert len(outcomes) == 3
    for _, returned, _, expected, _, left in outcomes:
        assert returned == expected and left == "0"
