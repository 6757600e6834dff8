"""The dense work of the host engine (host/dense.cpp) on the CPU."""
import ctypes as C
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "..", "nutrlan_b200", "csrc", "host", "dense.cpp")


def _preprocessed(tmp_path, *flags):
    """dense.cpp as the compiler's later stages see it, its includes empty."""
    for name in re.findall(r'#include [<"]([^>"]+)', open(SRC).read()):
        (tmp_path / name).write_text("")
    shutil.copy(SRC, tmp_path / "dense.cpp")
    return subprocess.run(["g++", "-E", "-P", "-nostdinc", "-I", str(tmp_path), *flags, str(tmp_path / "dense.cpp")],
                          check=True, capture_output=True, text=True).stdout


def test_no_x86_attribute_on_other_hosts(tmp_path):
    other = _preprocessed(tmp_path, "-U__x86_64__", "-U__i386__", "-D__aarch64__")
    assert "apply_sweep" in other and "avx" not in other
    if os.uname().machine == "x86_64":
        assert "avx2" in _preprocessed(tmp_path)


@pytest.fixture(scope="module")
def tridiag(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("dense") / "tridiag.so")
    inc = [f"-I{os.path.dirname(SRC)}", f"-I{os.path.join(HERE, '..', 'include')}"]
    subprocess.run(["g++", "-std=c++17", "-O3", "-fPIC", "-shared", *inc, os.path.join(HERE, "tridiag_vectors.cpp"), SRC,
                    "-o", so], check=True)
    return C.CDLL(so)


# Sizes on both sides of the 32 rows that are carried together; locked leading
# values; a coupling of zero in the middle (the matrix falls apart), graded
# entries, and entries whose squares leave the range of a double.
@pytest.mark.parametrize("kind", ["plain", "split", "graded", "huge", "tiny"])
@pytest.mark.parametrize("nd,locked,nrot", [(1, 0, 1), (2, 0, 2), (31, 0, 5), (32, 3, 1), (33, 0, 12), (64, 7, 20), (129, 0, 1)])
def test_vectors_of_the_tridiagonal(tridiag, nd, locked, nrot, kind):
    rng = np.random.default_rng(nd)
    a, b = rng.standard_normal(nd), 0.5 + rng.random(nd)
    if kind == "split":
        b[nd // 2] = 0.0
    elif kind == "graded":
        a, b = a * 10.0 ** -np.linspace(0, 12, nd), b * 10.0 ** -np.linspace(0, 12, nd)
    elif kind in ("huge", "tiny"):
        a, b = (v * (1e150 if kind == "huge" else 1e-150) for v in (a, b))
    n = nd - locked
    T = np.diag(a[locked:]) + np.diag(b[locked:nd - 1], 1) + np.diag(b[locked:nd - 1], -1)
    R = np.eye(n)
    R[:nrot, :nrot] = np.linalg.qr(rng.standard_normal((nrot, nrot)))[0]
    rot = np.ascontiguousarray(R[:nrot, :nrot].T)           # by columns
    lam, res, yy = np.zeros(nd), np.zeros(nd), np.zeros((n, n))
    P = lambda x: C.c_void_p(x.ctypes.data)
    assert tridiag.tridiag_vectors(nd, locked, P(a), P(b), nrot, P(rot), n, P(lam), P(res), P(yy)) == 0
    scale = np.abs(T).sum(axis=1).max()
    tol = 10 * n * np.finfo(float).eps                      # of QL with accumulated rotations
    np.testing.assert_allclose(lam[locked:] / scale, np.linalg.eigvalsh(T / scale), atol=tol)
    Y = R.T @ yy.T                                          # columns, the rotation taken back
    assert np.abs(Y.T @ Y - np.eye(n)).max() < tol
    assert np.abs((T / scale) @ Y - Y * (lam[locked:] / scale)).max() < tol
    np.testing.assert_allclose(res[locked:] / scale, b[nd - 1] / scale * np.abs(Y[-1]), atol=tol)
    np.testing.assert_array_equal(lam[:locked], a[:locked])
