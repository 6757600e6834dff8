"""Single-sweep Lanczos steps (kernels/sweep.cu) against the sequential
engine on the same operator and start vector.  Both run the reference's
recurrence and Gram-Schmidt (SRC/trlcore.c:1098-1116, 2913-3117) in FP64 and
differ in rounding only: Ritz values agree to 1e-12 relative (a few hundred
times the FP64 rounding of a dot product over these lengths), the counters
exactly."""
import numpy as np
import pytest

from nutrlan_b200 import operators as ops, DeviceOperator, solve

pytestmark = pytest.mark.gpu


def _operator(kind):
    if kind == "complex":
        return ops.peierls_2d(368, phi=1.0 / 16.0)      # 135,424 rows: the last tiles are partly padding
    return ops.anderson_3d(51, seed=5)                   # 132,651 rows


def _start(A):
    x0 = ops.start_vector(A.n)
    return x0 + 1j * ops.start_vector(A.n, seed=7) if np.iscomplexobj(A.val) else x0


# Basis sizes on both sides of one, two, four and eight column groups (16,
# 32, 64, 128) and past the 128 columns a sweep takes; the last with restarts.
@pytest.mark.parametrize("maxlan,maxmv", [(14, 14), (19, 19), (36, 36), (70, 70), (134, 134), (44, 120)])
@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("kind", ["real", "complex"])
def test_sweeps_match_sequential_steps(kind, bits, maxlan, maxmv, monkeypatch):
    A = _operator(kind)
    kw = dict(ned=5, maxlan=maxlan, tol=1e-13, restart=1, maxmv=maxmv, start=_start(A), basis_bits=bits, device=True)
    with DeviceOperator(A, fmt="sell") as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        swp = solve(op, **kw)
    assert seq.stats.speculative_steps == 0 and swp.stats.speculative_steps > 0
    assert swp.stats.kernel_launches < seq.stats.kernel_launches
    assert swp.stat == seq.stat == 0
    i, j = swp.info, seq.info
    assert (i.matvec, i.nloop, i.north, i.nrand) == (j.matvec, j.nloop, j.north, j.nrand)
    # A 32-bit basis stores each vector rounded to 2^-24: its Ritz values
    # follow the rounding decisions to the square of that times |A| / gap.
    np.testing.assert_allclose(swp.eval[:5], seq.eval[:5], rtol=1e-12 if bits == 64 else 1e-10)
    if bits == 64:
        k = swp.nec or 5
        V = swp.evec[:k]
        G = (V.conj() @ V.T).cpu().numpy()
        assert np.abs(G - np.eye(k)).max() < 1e-12      # Ritz vectors stay orthonormal


@pytest.mark.parametrize("bits", [64, 32])
def test_sweeps_fall_back_where_the_basis_is_exhausted(bits):
    """Six distinct eigenvalues: the Krylov space ends after six vectors, the
    steps that the sweeps took past it are rejected and taken again one at a
    time; every returned value is the smallest eigenvalue."""
    n = 1 << 17
    d = 1.0 + (np.arange(n) % 6)
    A = ops.CSR(n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), d)
    with DeviceOperator(A, fmt="sell") as op:
        r = solve(op, ned=3, maxlan=24, tol=1e-9, restart=1, maxmv=400, start=ops.start_vector(n), basis_bits=bits,
                  device=True)
    assert r.stat == 0 and r.nec >= 3
    assert r.stats.speculative_discarded > 0
    np.testing.assert_allclose(r.eval[:3], 1.0, rtol=1e-9)


def _band(n, width):
    """Symmetric matrix with `width` entries per inner row (and one row of
    10 * width, so that rows are uneven)."""
    import scipy.sparse as sp
    k = width // 2
    M = sp.diags([ops.start_vector(n, seed=17)] + [np.full(n - j, -1.0 / j) for j in range(1, k + 1)],
                 list(range(k + 1)), format="lil")
    M[7, 20:20 + 10 * width] = 0.01
    M = sp.triu(M).tocsr()
    M = (M + sp.triu(M, 1).T).tocsr()
    M.sort_indices()
    return ops.CSR(n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)


# The cooperative kernel over its range: one to many clusters, 32 to more than
# 512 rows per block, both operator forms, rows longer than a lane's batch and
# uneven ones, bases that stay in shared memory and ones that do not, restarts.
@pytest.mark.parametrize("case,fmt,maxlan,maxmv", [
    ("anderson7", "csr", 20, 60), ("anderson7", "sell", 20, 60), ("anderson12", "csr", 40, 110),
    ("anderson24", "sell", 30, 80), ("lattice253", "csr", 48, 100), ("lattice253", "sell", 150, 150),
    ("lattice340", "sell", 24, 60), ("peierls32", "csr", 24, 70), ("peierls32", "sell", 24, 70),
    ("peierls304", "sell", 60, 60), ("band24", "csr", 24, 60), ("band24", "sell", 24, 60)])
def test_cooperative_runs_match_sequential_steps(case, fmt, maxlan, maxmv, monkeypatch):
    size = int("".join(ch for ch in case if ch.isdigit()))
    if case.startswith("anderson"):
        A = ops.anderson_3d(size, seed=5)
    elif case.startswith("lattice"):
        A = ops.laplacian_2d(size, diag=2.0 * ops.uniform01(3, np.arange(size * size, dtype=np.uint64)))
    elif case.startswith("peierls"):
        A = ops.peierls_2d(size, phi=1.0 / 16.0)
    else:
        A = _band(5000, size)
    kw = dict(ned=4, maxlan=maxlan, tol=1e-13, restart=1, maxmv=maxmv, start=_start(A), device=True)
    with DeviceOperator(A, fmt=fmt) as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        coop = solve(op, **kw)
        again = solve(op, **kw)
    assert coop.stats.speculative_steps > 0 and coop.stats.kernel_launches < seq.stats.kernel_launches / 4
    assert coop.stat == seq.stat == 0
    i, j = coop.info, seq.info
    assert (i.matvec, i.nloop, i.north, i.nrand) == (j.matvec, j.nloop, j.north, j.nrand)
    np.testing.assert_allclose(coop.eval[:4], seq.eval[:4], rtol=1e-12, atol=1e-12 * np.abs(seq.eval[:4]).max())
    k = coop.nec or 4                                          # the pairs that come back
    V = coop.evec[:k]
    assert np.abs((V.conj() @ V.T).cpu().numpy() - np.eye(k)).max() < 1e-12
    np.testing.assert_array_equal(again.eval, coop.eval)      # the sums' order is fixed
    assert bool((again.evec[:k] == coop.evec[:k]).all())


def test_runs_on_badly_scaled_operators():
    """Entries of 1e-120: |r|^2 stays representable, r^H A r of unnormalised
    vectors would not; the solve takes such steps one at a time."""
    A = ops.anderson_3d(12, seed=5)
    small = ops.CSR(A.n, A.row_ptr, A.col, A.val * 1e-120)
    x0 = ops.start_vector(A.n)
    kw = dict(ned=4, maxlan=40, tol=1e-9, restart=1, maxmv=100000, start=x0, device=True)
    with DeviceOperator(A) as op, DeviceOperator(small) as ops_:
        r, s = solve(op, **kw), solve(ops_, **kw)
    assert r.nec >= 4 and s.nec >= 4
    np.testing.assert_allclose(s.eval[:4] * 1e120, r.eval[:4], rtol=1e-9)
