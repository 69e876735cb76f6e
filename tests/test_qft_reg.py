"""Register QFT passes (k_qft_reg), checked on the CPU: a host model of the kernel runs
every planned pass and must give the transform's definition (tests/cpp/test_qft_reg.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_qft_reg_passes(tmp_path):
    exe = str(tmp_path / "test_qft_reg")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "qpp_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_qft_reg.cpp"),
                    "-L", os.path.join(ROOT, "qpp_b200"), "-lqpp_b200",
                    f"-Wl,-rpath,{os.path.join(ROOT, 'qpp_b200')}", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "qft reg ok" in r.stdout
