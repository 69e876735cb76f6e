"""The wide blocks of the fused forms, checked on the CPU: their product is the
circuit (tests/cpp/test_fuse_wide.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_wide_blocks_are_the_circuit(tmp_path):
    exe = str(tmp_path / "test_fuse_wide")
    subprocess.run(["g++", "-std=c++17", "-O2",
                    "-I", os.path.join(ROOT, "qpp_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_fuse_wide.cpp"),
                    "-L", os.path.join(ROOT, "qpp_b200"), "-lqpp_b200",
                    f"-Wl,-rpath,{os.path.join(ROOT, 'qpp_b200')}", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "wide blocks ok" in r.stdout
