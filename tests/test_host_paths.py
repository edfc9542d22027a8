"""Host paths of the library over a fake CUDA runtime (tests/host): a posted
root that never comes, comes after a later commit took its mailbox slot, or
takes longer than the host spins for, posted elements that do, openings whose
copies or launch are refused, and the launches of a profiled commit."""
import os
import shutil
import subprocess

import pytest

HOST = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host")


@pytest.fixture(scope="module")
def host_paths(tmp_path_factory):
    from bitz_gb300 import build as B

    if not shutil.which("g++"):
        pytest.skip("no g++")
    B.build()
    objs = [os.path.join(B.BUILD, os.path.basename(s) + ".o") for s in B.sources()]
    if not all(map(os.path.exists, objs)):
        B.build(force=True)
    cuda = os.path.dirname(os.path.dirname(B.nvcc()))
    exe = str(tmp_path_factory.mktemp("host") / "host_paths")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-rdynamic", "-I", HOST, "-I", B.CSRC,
                        "-I", os.path.join(cuda, "include"),
                        os.path.join(HOST, "fake_cudart.cpp"),
                        os.path.join(HOST, "host_paths.cpp"), *objs, "-o", exe, "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("case", ["root_not_posted", "root_slot_reused", "root_slow",
                                  "root_stream_error", "elements_slow", "elements_not_posted",
                                  "opening_errors", "profile_is_the_commit"])
def test_host_path(host_paths, case):
    r = subprocess.run([host_paths, case], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
