"""The plan of the resident global step (csrc/resident.hpp), checked on the CPU by a C++ emulation
of its kernels (tests/cpp/resident_check.cpp): every row in one CTA, every halo slot filled by one
push per sweep, and the same bits as sweeps over the sliced ELL, for every number of lanes per
row and one to several groups and CTAs."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_resident_plan(tmp_path):
    exe = str(tmp_path / "resident_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "parallel_admm_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "resident_check.cpp"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip().endswith("ok")
