"""Sweeps of the trajectory kernel, checked on the CPU: the planned sweeps keep a
program's gates, order and noise steps (tests/cpp/test_sweeps.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sweeps_keep_the_program(tmp_path):
    exe = str(tmp_path / "test_sweeps")
    subprocess.run(["g++", "-std=c++17", "-O2",
                    "-I", os.path.join(ROOT, "qpp_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_sweeps.cpp"),
                    "-L", os.path.join(ROOT, "qpp_b200"), "-lqpp_b200",
                    f"-Wl,-rpath,{os.path.join(ROOT, 'qpp_b200')}", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "sweeps ok" in r.stdout
