"""The C entry points on a fake CUDA runtime (tests/cpp/fake_runtime.cpp), on the
CPU: what a failed call leaves behind, without a failing GPU, and what the calls that
share the workspace leave of the last render."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "jetshow_gb300", "csrc")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from jetshow_gb300 import build
    exe = str(tmp_path_factory.mktemp("fake") / "fake_runtime")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-I", CSRC, "-I", os.path.join(REPO, "include"), "-I",
                    os.path.join(build._cuda_home(), "include"), os.path.join(REPO, "tests", "cpp", "fake_runtime.cpp"),
                    os.path.join(CSRC, "jsh_capi.cpp"), os.path.join(CSRC, "jsh_host.cpp"), "-o", exe, "-lpthread"],
                   check=True)
    return exe


def run(exe, scenario):
    r = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_failed_launch_keeps_the_workspace_in_use(fake):
    run(fake, "error")


def test_last_stats_survive_other_calls(fake):
    run(fake, "statistics")


def test_segments_by_the_memory_there_is(fake):
    run(fake, "memory")
