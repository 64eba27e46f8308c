"""The shortlist's order of a catalog: every unit of 8 codes in exactly one part, ascending
within a part, no part more than the step less one times what comes before it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_parts_hold_every_unit_once(tmp_path):
    exe = str(tmp_path / "order")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "pure-sift_b200", "csrc"),
                    os.path.join(ROOT, "tests", "hamming_order.cpp"), "-o", exe], check=True)
    sizes = [0, 1, 7, 8, 9, 2047, 2048, 2049, 2056, 2057, 16376, 16384, 16385, 16392, 16393, 131072, 131073, 131081,
             65536, 65537, 300000, 1048577, 2000000, 2 ** 31 + 5, 2 ** 32 - 2] + [8 * n + r for n in range(257, 700) for r in (0, 3)]
    r = subprocess.run([exe, "check"] + [str(s) for s in sizes], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
