"""The choice between the two plans of fused blocks, checked on the CPU
(tests/cpp/test_fuse_best.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_cheaper_plan_is_taken(tmp_path):
    exe = str(tmp_path / "test_fuse_best")
    subprocess.run(["g++", "-std=c++17", "-O2",
                    "-I", os.path.join(ROOT, "qpp_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_fuse_best.cpp"),
                    "-L", os.path.join(ROOT, "qpp_b200"), "-lqpp_b200",
                    f"-Wl,-rpath,{os.path.join(ROOT, 'qpp_b200')}", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "best blocks ok" in r.stdout
