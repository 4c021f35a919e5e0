"""Plans the host makes for the kernels, checked without a GPU (tests/cpp/host_plans.cpp)."""
import os
import subprocess


def test_host_plans(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "host_plans")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", os.path.join(here, "cpp", "host_plans.cpp"), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout[:2000]
