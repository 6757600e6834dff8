"""Errors of CUDA calls in a run of Lanczos steps that is issued ahead of the
host's decisions reach the caller (CPU only: the library's object files
against a CUDA runtime that refuses what the test asks for; its kernels never
run, so the values of such a solve mean nothing)."""
import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

from nutrlan_b200._abi import MATVEC, TrlInfo, declare_common
from nutrlan_b200._lib import TrlxOptions

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(HERE, "..", "nutrlan_b200")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    objs = glob.glob(os.path.join(PKG, "_build", "kernels", "*.o")) + glob.glob(os.path.join(PKG, "_build", "host", "*.o"))
    if not objs or not os.path.exists(NVCC):
        pytest.skip("needs the build's object files and the CUDA headers")
    d = tmp_path_factory.mktemp("fake")
    rt, so, exports = str(d / "cudart.o"), str(d / "fake.so"), d / "exports.map"
    # (names of its own: the process may hold the library too)
    exports.write_text("{ global: trl*; ztrl*; fake_*; local: *; };")
    subprocess.run(["g++", "-fPIC", "-I", os.path.join(os.path.dirname(NVCC), "..", "include"),
                    "-c", os.path.join(HERE, "fake_cudart.cpp"), "-o", rt], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-Wl,--version-script=" + str(exports), rt, *objs,
                    "-ldl", "-lpthread", "-o", so], check=True)
    lib = C.CDLL(so)
    declare_common(lib)
    return lib


def _solve(fake, n, bits, launch_answer=0, sync_failures=0, maxlan=24):
    """info.stat of a solve on a diagonal operator; the number of runs asked for."""
    def var(name):
        return C.c_int.in_dll(fake, "fake_" + name)
    var("launches").value, var("launch_answer").value, var("sync_failures").value = 0, launch_answer, sync_failures
    rp, ci, va = np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n)
    op = C.c_void_p()
    P = lambda a: C.c_void_p(a.ctypes.data)
    assert fake.trlx_csr_create(n, P(rp), P(ci), P(va), 0, C.byref(op)) == 0
    info = TrlInfo()
    fake.trl_init_info(C.byref(info), n, maxlan, -1, 3, C.c_double(1e-9), 1, 40, None)
    info.verbose, info.mvparam = -1, op.value
    fake.trl_set_iguess(C.byref(info), 0, 1, 0, None)
    ev, vec, o = np.zeros(4), np.ones((4, n)), TrlxOptions(basis_bits=bits, refine=0)
    fake.trlx_trlan.restype = None
    fake.trlx_trlan(C.cast(fake.trlx_matvec, MATVEC), None, C.byref(info), n, 4, P(ev), P(vec), n, 0, None, C.byref(o))
    fake.trlx_operator_destroy(op)
    return info.stat, var("launches").value


# Cooperative runs (2000 rows), sweeps (2^17 rows), sweeps over a 32-bit basis.
@pytest.mark.parametrize("n,bits", [(2000, 64), (1 << 17, 64), (3000, 32)])
def test_error_in_a_run_is_the_solves_status(fake, n, bits):
    stat, runs = _solve(fake, n, bits, sync_failures=1)
    assert runs > 0 and stat == -1001


@pytest.mark.parametrize("n,bits", [(2000, 64), (1 << 17, 64), (3000, 32)])
def test_refused_launch_leaves_the_sequential_steps(fake, n, bits):
    stat, runs = _solve(fake, n, bits, launch_answer=701)
    assert runs > 0 and stat != -1001


def test_memory_for_runs_is_given_back_to_a_larger_solve(fake, monkeypatch):
    """The two vectors that a run of sweeps over a 32-bit basis goes back to are
    kept for the next solve, but not against its basis."""
    def size(name):
        return C.c_size_t.in_dll(fake, "fake_" + name)
    fake.trlx_release_workspace()
    size("peak").value = size("used").value
    monkeypatch.setenv("TRLX_SWEEP", "0")
    assert _solve(fake, 3000, 32, maxlan=60)[0] != -5
    need = size("peak").value               # without those vectors
    monkeypatch.delenv("TRLX_SWEEP")
    fake.trlx_release_workspace()
    assert _solve(fake, 3000, 32)[1] > 0    # the smaller solve takes sweeps
    size("limit").value = need
    try:
        assert _solve(fake, 3000, 32, maxlan=60)[0] != -5
    finally:
        size("limit").value = 0
