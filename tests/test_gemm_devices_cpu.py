"""The GEMM raises its kernels' shared-memory limit on every device it is launched on: its host code
against a fake CUDA runtime with two devices."""
import os
import subprocess

from conftest import ROOT


def test_shared_memory_limit_is_raised_on_every_device(tmp_path):
    from tdp1375_b200 import build
    build.build()
    exe = str(tmp_path / "gemm_devices")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "host", "gemm_devices.cpp"),
                    os.path.join(build.OBJ, "mlp_gemm.cu.o"), "-lpthread", "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
