"""The guard of settings that belong to a device (gb_once.h), built for the host
with a cudaGetDevice of its own."""
import os
import subprocess

from slothdb_gb300 import build


def test_once_per_device(tmp_path):
    exe = str(tmp_path / "once_per_device")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", build.CSRC, "-isystem", os.path.join(cuda, "include"),
                    os.path.join(build.ROOT, "tests", "cpp", "once_per_device.cpp"), "-o", exe], check=True)
    subprocess.run([exe], check=True)
