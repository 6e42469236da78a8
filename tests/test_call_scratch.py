"""The device scratch kept between calls is bounded and given back however a call ends (over a fake of the CUDA
runtime's allocation calls)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scratch_is_given_back(tmp_path):
    exe = str(tmp_path / "call_scratch")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{cuda}/include", os.path.join(ROOT, "tests", "cpp", "call_scratch.cpp"),
                    "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
