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
        V = swp.evec[:5]
        G = (V.conj() @ V.T).cpu().numpy()
        assert np.abs(G - np.eye(5)).max() < 1e-12      # Ritz vectors stay orthonormal


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
