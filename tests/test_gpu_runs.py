"""Runs of Lanczos steps that are issued ahead of the host's decisions, where
they go wrong or do not apply: the solve goes on with the sequential steps
(trl_orth's decisions, SRC/trlcore.c:2913-3117) and gives what those give."""
import ctypes as C

import numpy as np
import pytest

from nutrlan_b200 import operators as ops, DeviceOperator, solve

pytestmark = pytest.mark.gpu


def _start(A):
    x0 = ops.start_vector(A.n)
    return x0 + 1j * ops.start_vector(A.n, seed=7) if np.iscomplexobj(A.val) else x0


def _same(a, b, k):
    assert a.stat == b.stat == 0
    i, j = a.info, b.info
    assert (i.matvec, i.nloop, i.north, i.nrand) == (j.matvec, j.nloop, j.north, j.nrand)
    np.testing.assert_allclose(a.eval[:k], b.eval[:k], rtol=1e-12, atol=1e-12 * np.abs(b.eval[:k]).max())


# One cluster and many, real and complex, a run of one step and longer ones.
@pytest.mark.parametrize("A,maxlan,maxmv", [
    (ops.anderson_3d(7, seed=5), 20, 60), (ops.anderson_3d(24, seed=5), 30, 80), (ops.laplacian_2d(253), 40, 90),
    (ops.peierls_2d(64, phi=1.0 / 16.0), 24, 70)])
@pytest.mark.parametrize("polls", ["0", "2"])
def test_cooperative_run_whose_barrier_gives_up_is_not_used(A, maxlan, maxmv, polls, monkeypatch):
    """The grid barrier's wait cut to nothing: blocks go on without the others'
    sums, the run is reported as failed, and none of its steps is taken."""
    kw = dict(ned=4, maxlan=maxlan, tol=1e-13, restart=1, maxmv=maxmv, start=_start(A), device=True)
    with DeviceOperator(A, fmt="sell") as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        monkeypatch.setenv("TRLX_COOP_POLLS", polls)
        cut = solve(op, **kw)
        monkeypatch.delenv("TRLX_COOP_POLLS")
        full = solve(op, **kw)
    assert cut.stats.speculative_discarded > 0
    assert full.stats.speculative_discarded == 0 and full.stats.speculative_steps > 0
    _same(cut, seq, 4)
    _same(full, seq, 4)


def _uneven(n, cplx):
    """A grid Laplacian with every eleventh row coupled to 12 more, so that a
    SELL operator of sorted rows keeps them in another order."""
    import scipy.sparse as sp
    L = int(n ** 0.5)
    A = ops.laplacian_2d(L, diag=2.0 * ops.uniform01(3, np.arange(L * L, dtype=np.uint64))).to_scipy().tolil()
    for r in range(0, L * L, 11):
        for q in range(1, 13):
            c = (r + 37 * q) % (L * L)
            A[r, c] = A[c, r] = -0.01 * q
    A = A.tocsr()
    A.sort_indices()
    if cplx:
        U = sp.triu(A, 1) * np.exp(0.3j)
        A = (U + U.conj().T + sp.diags(A.diagonal())).tocsr()
        A.sort_indices()
    return ops.CSR(L * L, A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data)


# Row-sorted SELL operators, which the cooperative kernel does not take, real
# and complex.
@pytest.mark.parametrize("n,cplx", [(30 * 30, False), (100 * 100, False), (60 * 60, True)])
def test_operators_the_cooperative_kernel_refuses(n, cplx, monkeypatch):
    """After a restart the first step couples to all kept vectors; no run that
    knows only the last two is started with it, to be thrown away."""
    A = _uneven(n, cplx)
    kw = dict(ned=4, maxlan=30, tol=1e-10, restart=1, maxmv=400, start=_start(A), device=True)
    with DeviceOperator(A, fmt="sell", sigma=64) as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        got = solve(op, **kw)
    assert seq.info.nloop > 3
    assert got.stats.speculative_steps > 0 and got.stats.speculative_discarded == 0
    _same(got, seq, 4)


def _hubs(n, width, hubs, cplx=False):
    """A band matrix of `width` entries per inner row; row r has about `deg`
    entries more for each (r, deg) of `hubs`."""
    import scipy.sparse as sp
    k = width // 2
    U = sp.diags([np.full(n - j, -1.0 / j) for j in range(1, k + 1)], list(range(1, k + 1)), shape=(n, n)).tocoo()
    at, to = [U.row], [U.col]
    v = [U.data]
    for r, deg in hubs:
        c = np.setdiff1d(np.linspace(0, n - 1, deg).astype(np.int64), [r])
        at.append(np.minimum(r, c)), to.append(np.maximum(r, c)), v.append(np.full(c.size, -0.01))
    U = sp.coo_matrix((np.concatenate(v), (np.concatenate(at), np.concatenate(to))), shape=(n, n)).tocsr()
    if cplx:
        U = U * np.exp(0.3j)
    A = (U + U.conj().T + sp.diags(4.0 * ops.uniform01(3, np.arange(n, dtype=np.uint64)))).tocsr()
    A.sort_indices()
    return ops.CSR(n, A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data)


# Rows on both sides of 32 entries (one lane a row, a warp above), the first
# and the last of all, many of them in one block; two and sixteen lanes a row;
# entries kept in shared memory and not.
@pytest.mark.parametrize("fmt", ["csr", "sell"])
@pytest.mark.parametrize("n,width,hubs,cplx", [
    (3001, 5, [(0, 27), (100, 28), (101, 29), (3000, 300)], False), (5000, 5, [(r, 40) for r in range(64, 200)], False),
    (40000, 5, [(39999, 9000), (7, 20000)], False), (5000, 13, [(9, 59), (10, 61), (4999, 2500)], False),
    (3000, 91, [(0, 2900), (1, 500)], False), (5000, 5, [(0, 31), (2500, 2000), (2501, 5000)], True)])
def test_cooperative_runs_on_long_rows(n, width, hubs, cplx, fmt, monkeypatch):
    A = _hubs(n, width, hubs, cplx)
    kw = dict(ned=4, maxlan=24, tol=1e-13, restart=1, maxmv=60, start=_start(A), device=True)
    with DeviceOperator(A, fmt=fmt) as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        coop = solve(op, **kw)
        again = solve(op, **kw)
    assert coop.stats.speculative_steps > 0 and coop.stats.kernel_launches < seq.stats.kernel_launches / 4
    _same(coop, seq, 4)
    np.testing.assert_array_equal(again.eval, coop.eval)


@pytest.mark.parametrize("cplx", [False, True])
def test_long_row_is_not_left_to_a_few_lanes(cplx, monkeypatch):
    """One row of 3000 entries: a cooperative run takes no longer than the
    discrete kernels, which give every row eight lanes."""
    A = _hubs(30000, 5, [(15000, 3000)], cplx)
    kw = dict(ned=4, maxlan=40, tol=1e-13, restart=1, maxmv=80, start=_start(A), device=True)

    def best(op):
        return min(solve(op, **kw).stats.seconds_total for _ in range(5))
    with DeviceOperator(A, fmt="csr") as op:
        coop = best(op)
        monkeypatch.setenv("TRLX_COOP", "0")
        discrete = best(op)
    assert coop < discrete


# A 32-bit basis of few rows: the rounding of the stored vectors makes a second
# pass necessary every few steps.
@pytest.mark.parametrize("L", [6, 8, 10])
def test_runs_shorten_where_steps_are_rejected(L, monkeypatch):
    A = ops.anderson_3d(L, seed=5)
    kw = dict(ned=6, maxlan=48, tol=1e-13, restart=1, maxmv=150, start=_start(A), basis_bits=32, device=True)
    with DeviceOperator(A, fmt="csr") as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        got = solve(op, **kw)
    assert seq.info.north > 0 and got.stat == seq.stat == 0
    assert got.stats.speculative_discarded <= 150 // 2      # no more than half the solve's steps
    np.testing.assert_allclose(got.eval[:6], seq.eval[:6], rtol=1e-10)


def _random(n, per, cplx=False, longest=0):
    """About `per` entries a row in random columns; row 0 with `longest`."""
    import scipy.sparse as sp
    rng = np.random.default_rng(1)
    m = n * (per - 1) // 2
    i, j, v = rng.integers(0, n, m), rng.integers(0, n, m), rng.standard_normal(m)
    if longest:
        c = rng.choice(np.arange(1, n), longest, replace=False)
        i, j, v = np.concatenate([i, np.zeros_like(c)]), np.concatenate([j, c]), np.concatenate([v, np.full(longest, -0.01)])
    U = sp.triu(sp.coo_matrix((np.concatenate([v, v]), (np.concatenate([i, j]), np.concatenate([j, i]))), shape=(n, n)).tocsr(), 1)
    if cplx:
        U = U * np.exp(0.3j)
    A = (U + U.conj().T + sp.diags(rng.standard_normal(n))).tocsr()
    A.sort_indices()
    return ops.CSR(n, A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data)


# Operators on both sides of the lines between cooperative runs (one launch for
# many steps) and sweeps (two a step): doubles to gather in a product, and the
# longest row against them.
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("n,per,cplx,longest,fmt,one", [
    (30000, 49, False, 0, "csr", True), (30000, 53, False, 0, "csr", False), (15000, 49, True, 0, "csr", True),
    (15000, 53, True, 0, "csr", False), (30000, 65, False, 6000, "csr", True), (30000, 65, False, 0, "sell", False),
    (30000, 65, False, 900, "sell", True)])
def test_steps_of_operators_with_many_entries(n, per, cplx, longest, fmt, one, device, monkeypatch):
    A = _random(n, per, cplx, longest)
    kw = dict(ned=4, maxlan=24, tol=1e-13, restart=1, maxmv=60, start=_start(A), device=True)
    with DeviceOperator(A, fmt=fmt) as op:
        if device:      # the same operator from arrays on the device
            import torch
            arrays = [torch.as_tensor(a).cuda() for a in (A.row_ptr, A.col, A.val)]
            op.close()
            create = getattr(op.lib, f"trlx_{op.fmt}_create")
            args = [n, *(a.data_ptr() for a in arrays)] + ([1] if fmt == "sell" else [])
            assert create(*args, 1, C.byref(op.handle)) == 0
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        got = solve(op, **kw)
    assert got.stats.speculative_steps > 0 and got.stats.speculative_discarded == 0
    assert (got.stats.kernel_launches < 60) == one
    _same(got, seq, 4)


@pytest.mark.parametrize("fmt", ["csr", "sell"])
def test_many_entries_are_not_gathered_twice(fmt, monkeypatch):
    """65536 rows of 65 entries: steps take no longer than with the discrete
    kernels."""
    A = _random(65536, 65)
    kw = dict(ned=4, maxlan=40, tol=1e-13, restart=1, maxmv=80, start=_start(A), device=True)

    def best(op):
        return min(solve(op, **kw).stats.seconds_total for _ in range(5))
    with DeviceOperator(A, fmt=fmt) as op:
        got = best(op)
        monkeypatch.setenv("TRLX_COOP", "0")
        monkeypatch.setenv("TRLX_SWEEP", "0")
        discrete = best(op)
    assert got < discrete


# Rows that are no multiple of 256: what a rejected run leaves in the padding
# rows of the columns (its scale is no number) does not reach a result.
@pytest.mark.parametrize("n,bits", [((1 << 17) + 77, 64), (3001, 64), (5003, 32)])
@pytest.mark.parametrize("fmt", ["csr", "sell"])
def test_exhausted_basis_with_padding_rows(n, bits, fmt, monkeypatch):
    A = ops.CSR(n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), 1.0 + (np.arange(n) % 6))
    kw = dict(ned=3, maxlan=24, tol=1e-9, restart=1, maxmv=400, start=ops.start_vector(n), basis_bits=bits, device=True)
    with DeviceOperator(A, fmt=fmt) as op:
        r = solve(op, **kw)
        B = ops.anderson_3d(17, seed=5)             # the same workspace after it
        kw.update(start=_start(B), maxmv=60, maxlan=24, tol=1e-13)
        with DeviceOperator(B, fmt=fmt) as op2:
            after = solve(op2, **kw)
            monkeypatch.setenv("TRLX_SPECULATE", "0")
            seq = solve(op2, **kw)
    assert r.stat == 0 and r.nec >= 3 and r.stats.speculative_discarded > 0
    np.testing.assert_allclose(r.eval[:3], 1.0, rtol=1e-9)
    np.testing.assert_allclose(after.eval[:3], seq.eval[:3], rtol=1e-12 if bits == 64 else 1e-10)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 12])
@pytest.mark.parametrize("bits", [64, 32])
def test_runs_on_the_smallest_problems(n, bits, monkeypatch):
    """The basis spans the whole space before a run ends."""
    import scipy.sparse as sp
    M = sp.diags([np.arange(1.0, n + 1), np.full(n - 1, -0.5), np.full(n - 1, -0.5)], [0, 1, -1], format="csr")
    M.sort_indices()
    A = ops.CSR(n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)
    kw = dict(ned=1, maxlan=max(n, 3), tol=1e-10, restart=1, maxmv=60, start=np.ones(n), basis_bits=bits, device=True)
    with DeviceOperator(A) as op:
        monkeypatch.setenv("TRLX_SPECULATE", "0")
        seq = solve(op, **kw)
        monkeypatch.delenv("TRLX_SPECULATE")
        got = solve(op, **kw)
    assert got.stat == seq.stat and got.nec == seq.nec
    if seq.nec:
        np.testing.assert_allclose(got.eval[:1], seq.eval[:1], rtol=1e-9)
