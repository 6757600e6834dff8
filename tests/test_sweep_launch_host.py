"""A sweep that CUDA did not launch is reported to the engine, which must not
read its log (CPU only: the library's object file against a CUDA runtime that
answers what the test asks for)."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(HERE, "..", "nutrlan_b200")
OBJ = os.path.join(PKG, "_build", "kernels", "sweep.o")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(OBJ) or not os.path.exists(NVCC):
        pytest.skip("needs the build's object files and nvcc")
    d = tmp_path_factory.mktemp("fake")
    call, rt, so = str(d / "call.o"), str(d / "cudart.o"), str(d / "fake.so")
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(PKG, "csrc"), "-c", os.path.join(HERE, "sweep_launch.cu"), "-o", call],
                   check=True)
    subprocess.run(["g++", "-fPIC", "-I", os.path.join(os.path.dirname(NVCC), "..", "include"),
                    "-c", os.path.join(HERE, "fake_cudart.cpp"), "-o", rt], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", call, rt, OBJ, "-o", so], check=True)
    return C.CDLL(so)


def test_sweep_reports_a_failed_launch(fake):
    def status(device, attribute, launch):
        for name, v in (("device", device), ("attribute_answer", attribute), ("launch_answer", launch)):
            C.c_int.in_dll(fake, "fake_" + name).value = v
        return fake.sweep_status()

    launches = C.c_int.in_dll(fake, "fake_launches")
    # (each device is asked for its attributes once)
    assert status(0, 1, 0) != 0 and launches.value == 0      # the shared memory was refused
    assert status(1, 0, 0) == 0 and launches.value == 1
    assert status(1, 0, 701) != 0 and launches.value == 2    # the launch was refused
    assert status(1, 0, 0) == 0 and launches.value == 3
