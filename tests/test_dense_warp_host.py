"""The dense routines that one warp of a batched problem runs at its restarts
(kernels/dense_warp.cuh), on the CPU with the lanes run one after the other
between their __syncwarp() calls, in both orders: a lane that reads what
another one writes without a __syncwarp() between gives other results.
Eigenvalues and vectors against numpy's symmetric solver."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "nutrlan_b200", "csrc")


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("warp") / "warp_lanes.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(CSRC, "kernels"),
                    os.path.join(HERE, "warp_lanes.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.warp_ws_doubles.restype = C.c_long
    return lib


def P(a):
    return C.c_void_p(a.ctypes.data)


def _problem(nd, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(nd), np.abs(rng.standard_normal(nd)) + 0.01


# Up to the largest projected problem (66), on both sides of one and two rows a lane.
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("nd,locked", [(1, 0), (2, 0), (3, 1), (24, 0), (32, 5), (33, 0), (64, 3), (66, 0)])
def test_eigenvalues_whatever_the_order_of_the_lanes(lanes, nd, locked, order):
    a, b = _problem(nd, 100 * nd + locked)
    m = nd - locked
    T = np.diag(a[locked:]) + np.diag(b[locked:nd - 1], 1) + np.diag(b[locked:nd - 1], -1)
    w, Q = np.linalg.eigh(T)
    # A QL solve is backward stable: a few roundings of |T| per rotation sweep.
    tol = 1e-15 * nd * (1.0 + np.abs(T).max())
    for vectors in (0, 1):
        lam, res = np.zeros(nd), np.zeros(nd)
        ws = np.zeros(lanes.warp_ws_doubles(nd))
        assert lanes.warp_get_eval(order, nd, locked, P(a), P(b), P(lam), P(res), vectors, P(ws)) == 0
        np.testing.assert_array_equal(lam[:locked], a[:locked])
        np.testing.assert_allclose(lam[locked:], w, atol=tol)
        if vectors:
            Z = ws[2 * m:2 * m + m * m].reshape(m, m)      # one eigenvector per row
            assert np.abs(Z @ Z.T - np.eye(m)).max() < tol
            assert np.abs(Z @ T - ws[:m, None] * Z).max() < 10 * tol


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("nd,kept", [(2, 1), (24, 12), (33, 16), (64, 40)])
def test_arrowhead_vectors_whatever_the_order_of_the_lanes(lanes, nd, kept, order):
    a, b = _problem(nd, nd + kept)
    H = np.diag(a)
    H[:kept, kept] = H[kept, :kept] = b[:kept]
    for i in range(kept, nd - 1):
        H[i, i + 1] = H[i + 1, i] = b[i]
    w = np.linalg.eigvalsh(H)
    n = max(1, nd // 2)
    al, yy = a.copy(), np.zeros((n, nd))
    ws = np.zeros(lanes.warp_ws_doubles(nd))
    assert lanes.warp_get_tvec_a(order, nd, kept, P(al), P(b), n, P(w[:n].copy()), P(yy), P(ws)) == 0
    tol = 1e-15 * nd * (1.0 + np.abs(H).max())
    np.testing.assert_allclose(al[:n], w[:n], atol=tol)
    assert np.abs(yy @ yy.T - np.eye(n)).max() < tol
    assert np.abs(yy @ H - al[:n, None] * yy).max() < 10 * tol
