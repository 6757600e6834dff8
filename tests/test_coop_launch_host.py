"""launch_coop from two threads, the second while the first one asks what the
device holds (CPU only: the kernel's object file against a CUDA runtime that
lets the test in between)."""
import ctypes as C
import os
import shutil
import subprocess
import threading

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(HERE, "..", "nutrlan_b200")
OBJ = os.path.join(PKG, "_build", "kernels", "coop.o")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(OBJ) or not os.path.exists(NVCC):
        pytest.skip("needs the build's object files and nvcc")
    d = tmp_path_factory.mktemp("fake")
    call, rt, so, exports = str(d / "call.o"), str(d / "cudart.o"), str(d / "fake.so"), d / "exports.map"
    exports.write_text("{ global: coop_status; fake_*; local: *; };")
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(PKG, "csrc"), "-c", os.path.join(HERE, "coop_launch.cu"), "-o", call], check=True)
    subprocess.run(["g++", "-fPIC", "-I", os.path.join(os.path.dirname(NVCC), "..", "include"),
                    "-c", os.path.join(HERE, "fake_cudart.cpp"), "-o", rt], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-Wl,--version-script=" + str(exports),
                    call, rt, OBJ, "-o", so], check=True)
    return C.CDLL(so)


def test_second_thread_during_the_first_ones_setup(fake):
    got, second = {}, []

    @C.CFUNCTYPE(None, C.c_int)
    def between(call):
        if call == 2:                       # clusters of 8 are known, those of 4 not yet
            t = threading.Thread(target=lambda: got.update(second=fake.coop_status(1 << 16)))
            t.start()
            t.join(0.5)                     # it is done, or waits for this thread
            second.append(t)

    C.c_void_p.in_dll(fake, "fake_on_occupancy").value = C.cast(between, C.c_void_p).value
    got["first"] = fake.coop_status(1 << 16)
    second[0].join()
    assert got == {"first": 0, "second": 0}
