"""Host side of the Hamming shortlist entries, on a stand-in for the CUDA runtime
(topk_host.cpp): what the callers are told when something on the device fails."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("topk") / "topk_host")
    csrc = os.path.join(ROOT, "pure-sift_b200", "csrc")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(cuda, "include"),
                    "-I", os.path.join(ROOT, "include"), "-I", csrc,
                    "-x", "c++", os.path.join(ROOT, "tests", "topk_host.cpp"), os.path.join(csrc, "catalog_api.cu"),
                    os.path.join(csrc, "ctx.cu"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["timeout", "memory"])
def test_failures_reach_the_caller(harness, scenario):
    r = subprocess.run([harness, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
