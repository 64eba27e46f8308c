"""Host side of the RANSAC entries, on a stand-in for the CUDA runtime (ransac_host.cpp): the
workspace holds what the kernel uses and no more."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_workspace_of_a_match_set(tmp_path):
    exe = str(tmp_path / "ransac_host")
    csrc = os.path.join(ROOT, "pure-sift_b200", "csrc")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(cuda, "include"),
                    "-I", os.path.join(ROOT, "include"), "-I", csrc,
                    "-x", "c++", os.path.join(ROOT, "tests", "ransac_host.cpp"), os.path.join(csrc, "ransac_api.cu"),
                    os.path.join(csrc, "ctx.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
