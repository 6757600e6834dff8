"""Runs of Lanczos steps that are issued ahead of the host's decisions, where
they go wrong or do not apply: the solve goes on with the sequential steps
(trl_orth's decisions, SRC/trlcore.c:2913-3117) and gives what those give."""
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
