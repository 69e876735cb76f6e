"""Register tile passes, checked on the CPU: the planned programs
run on a host model of the kernel give the gate-by-gate result
(tests/cpp/test_reg_tiles.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_register_tile_programs_match_gate_by_gate(tmp_path):
    exe = str(tmp_path / "test_reg_tiles")
    subprocess.run(["g++", "-std=c++17", "-O2",
                    "-I", os.path.join(ROOT, "qpp_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_reg_tiles.cpp"),
                    "-L", os.path.join(ROOT, "qpp_b200"), "-lqpp_b200",
                    f"-Wl,-rpath,{os.path.join(ROOT, 'qpp_b200')}", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "reg tiles ok" in r.stdout
