"""The work a user of this package has it do, as cases that can be timed and checked.

Both kinds go through the entry points of the Python package:

* ``solve``: ``solve()``, the thick-restart Lanczos path, on a
  ``DeviceOperator`` or on the caller's own operator callback: lattice
  operators from a thousand rows (launch latency) to 256^3 rows (memory
  bandwidth), real and complex, 64- and 32-bit basis storage, eigenvectors
  left on the device or returned to the host.  A pass is bounded by ``maxmv``
  to whole restart cycles, so that a pass is the same work whatever the start
  vector.
* ``batch``: ``Batch.solve()``, many small problems of uneven size solved to
  convergence in one launch.

Inputs are made on the GPU from the seed alone.
"""
import ctypes as C
import math

import numpy as np
import torch

from nutrlan_b200 import MATVEC, DeviceOperator, operators, solve
from nutrlan_b200.batched import Batch

DEV = "cuda"


def listed():
    return [
        # The smallest calls: a 12^3 lattice, eigenvectors to host memory, a
        # few restarts.  Launches, host round trips and the small dense work
        # of the restarts are all there is.
        dict(name="anderson12_host", kind="solve", family="anderson", L=12, ned=8, maxlan=40, cycles=3, bits=64,
             fmt="csr", host=True),
        # A 128^2 grid, smallest 10, basis 64: the size of the package's
        # first example, several restarts.
        dict(name="lattice128", kind="solve", family="lattice", L=128, ned=10, maxlan=64, cycles=4, bits=64,
             fmt="csr", host=False),
        # One 256^2 potential-well operator, smallest 16, basis 48, tuned
        # operator: the solves of a dataset of potentials.
        dict(name="wells256_auto", kind="solve", family="wells", L=256, ned=16, maxlan=48, cycles=3, bits=64,
             fmt="auto", host=False),
        # Complex Hermitian 256^2 lattice, smallest 8, eigenvectors to host.
        dict(name="peierls256_host", kind="solve", family="peierls", L=256, ned=8, maxlan=48, cycles=2, bits=64,
             fmt="csr", host=True),
        # The caller's own operator (a matvec callback on device pointers), as
        # programs written for the reference library have.
        dict(name="lattice300_callback", kind="solve", family="lattice", L=300, ned=10, maxlan=64, cycles=2, bits=64,
             fmt="callback", host=False),
        # 64^3: a basis of a few hundred MB, between latency and bandwidth.
        dict(name="anderson64", kind="solve", family="anderson", L=64, ned=32, maxlan=128, cycles=2, bits=64,
             fmt="sell", host=False),
        # 32-bit basis storage, odd row count.
        dict(name="anderson101_fp32", kind="solve", family="anderson", L=101, ned=12, maxlan=96, cycles=2, bits=32,
             fmt="sell", host=False),
        # Complex Hermitian 1024^2 lattice, complex128 basis.
        dict(name="peierls1024", kind="solve", family="peierls", L=1024, ned=16, maxlan=96, cycles=2, bits=64,
             fmt="sell", host=False),
        # Complex Hermitian 2048^2 lattice, complex64 basis, tuned operator.
        dict(name="peierls2048_c64", kind="solve", family="peierls", L=2048, ned=16, maxlan=96, cycles=1, bits=32,
             fmt="auto", host=False),
        # The benchmark's call: 256^3, smallest 32, basis 128, tuned operator.
        dict(name="anderson256", kind="solve", family="anderson", L=256, ned=32, maxlan=128, cycles=1, bits=64,
             fmt="auto", host=False),
        # A few dozen small problems: fewer than the GPU has room for.
        dict(name="batch40", kind="batch", problems=40, lo=20, hi=64, ned=8, maxlan=32),
        # A few hundred problems of the benchmark's size range.
        dict(name="batch400", kind="batch", problems=400, lo=48, hi=160, ned=8, maxlan=32),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.2:
        lo = rng.randint(16, 64)
        return dict(kind="batch", problems=_logint(rng, 16, 400), lo=lo, hi=lo + rng.randint(8, 96),
                    ned=rng.randint(4, 10), maxlan=rng.choice([24, 28, 32, 40]))
    family = rng.choice(["anderson", "anderson", "lattice", "wells", "peierls"])
    if family == "anderson":
        L = _logint(rng, 12, 200)
    elif family == "peierls":
        L = 16 * _logint(rng, 2, 96)
    else:
        L = _logint(rng, 40, 1500)
    ned = rng.randint(4, 32)
    maxlan = max(2 * ned + 8, rng.randint(24, 128))
    return dict(kind="solve", family=family, L=L, ned=ned, maxlan=maxlan, cycles=rng.randint(1, 2),
                bits=rng.choice([64, 64, 32]), fmt=rng.choice(["csr", "csr", "sell", "sell", "auto", "auto", "callback"]),
                host=rng.random() < 0.3)


# ---- inputs -----------------------------------------------------------------
def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEV, dtype=torch.float64)


def _wells(gen, B, H, W, nwells=8):
    """B potentials on an H x W grid, each a sum of Gaussian wells."""
    u = _rand(gen, B, nwells, 4)
    y = torch.arange(H, device=DEV, dtype=torch.float64)[None, :, None]
    x = torch.arange(W, device=DEV, dtype=torch.float64)[None, None, :]
    V = torch.zeros(B, H, W, device=DEV, dtype=torch.float64)
    for k in range(nwells):
        cx, cy, w, d = (u[:, k, i].reshape(B, 1, 1) for i in range(4))
        r2 = (x - cx * W) ** 2 + (y - cy * H) ** 2
        V -= (5.0 + 45.0 * d) * torch.exp(-r2 / (2.0 * (4.0 + 20.0 * w) ** 2))
    return V


def _entries(case, gen):
    """(n, columns (n, k), values (n, k), inside (n, k) or None) of the operator, on the device."""
    L, family = case["L"], case["family"]
    n = L ** 3 if family == "anderson" else L * L
    i = torch.arange(n, device=DEV)
    x, y = i % L, (i // L) % L
    if family == "anderson":  # periodic 7-point hopping, random diagonal of width 4
        z = i // (L * L)
        nb = [(x + 1) % L + L * (y + L * z), (x - 1) % L + L * (y + L * z), x + L * ((y + 1) % L + L * z),
              x + L * ((y - 1) % L + L * z), x + L * (y + L * ((z + 1) % L)), x + L * (y + L * ((z - 1) % L))]
        cols = torch.stack([i] + nb, dim=1)
        vals = torch.full((n, 7), -1.0, device=DEV, dtype=torch.float64)
        vals[:, 0] = 4.0 * (_rand(gen, n) - 0.5)
        return n, cols, vals, None
    if family == "peierls":  # periodic, flux 1/16 per plaquette, random diagonal of width 2
        ph = torch.polar(torch.ones(n, device=DEV, dtype=torch.float64), (2.0 * math.pi / 16.0) * (x % 16).double())
        cols = torch.stack([i, (x + 1) % L + L * y, (x - 1) % L + L * y, x + L * ((y + 1) % L), x + L * ((y - 1) % L)],
                           dim=1)
        vals = torch.full((n, 5), -1.0, device=DEV, dtype=torch.complex128)
        vals[:, 0] = 2.0 * (_rand(gen, n) - 0.5)
        vals[:, 3] = -ph.conj()
        vals[:, 4] = -ph
        return n, cols, vals, None
    # 5-point Dirichlet Laplacian plus a diagonal potential.
    d = 2.0 * _rand(gen, n) if family == "lattice" else _wells(gen, 1, L, L).reshape(-1)
    cols = torch.stack([i, i - 1, i + 1, i - L, i + L], dim=1)
    vals = torch.full((n, 5), -1.0, device=DEV, dtype=torch.float64)
    vals[:, 0] = 4.0 + d
    inside = torch.stack([x >= 0, x > 0, x < L - 1, y > 0, y < L - 1], dim=1)
    return n, cols, vals, inside


def _csr(n, cols, vals, inside):
    """Rows sorted by column, as the package's CSR (host arrays)."""
    k = cols.shape[1]
    if inside is not None:
        cols = torch.where(inside, cols, torch.full_like(cols, n))
    cols, order = torch.sort(cols, dim=1)
    vals = torch.gather(vals, 1, order)
    if inside is None:
        row_ptr = torch.arange(0, k * n + 1, k, device=DEV)
        cols, vals = cols.reshape(-1), vals.reshape(-1)
    else:
        keep = cols < n
        row_ptr = torch.zeros(n + 1, device=DEV, dtype=torch.int64)
        row_ptr[1:] = keep.sum(dim=1).cumsum(0)
        cols, vals = cols[keep], vals[keep]
    return operators.CSR(n, row_ptr.cpu().numpy(), cols.to(torch.int32).cpu().numpy(), vals.cpu().numpy())


def _start(gen, n, cplx):
    v = 2.0 * _rand(gen, n) - 1.0
    return torch.complex(v, 2.0 * _rand(gen, n) - 1.0) if cplx else v


def _batch_inputs(case, gen):
    u = _rand(gen, case["problems"]).cpu().numpy()
    Ls = (case["lo"] + np.floor(u * (case["hi"] - case["lo"] + 1))).astype(np.int32)
    return Ls, [(2.0 * _rand(gen, int(L) * int(L))).cpu().numpy() for L in Ls]


class _Callback:
    """The caller's own operator: a matvec on device pointers that the solver
    knows nothing about (here it forwards to the library's product)."""

    def __init__(self, op):
        f = op.lib.trlx_zmatvec if op.complex else op.lib.trlx_matvec
        f.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_void_p]
        f.restype = None
        self.op, self.n, self.complex, self.handle = op, op.n, op.complex, C.c_void_p(None)
        self.applier = MATVEC(lambda nrow, ncol, x, ldx, y, ldy, p: f(nrow, ncol, x, ldx, y, ldy, op.handle))


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    s = {"case": case}
    if case["kind"] == "solve":
        A = _csr(*_entries(case, gen))
        if case["fmt"] == "callback":
            s["op"] = _Callback(DeviceOperator(A, fmt="csr"))
        else:
            s["op"] = DeviceOperator(A, fmt=case["fmt"], maxlan=case["maxlan"])
        s["start"] = _start(gen, A.n, s["op"].complex)
        if _host(case):
            s["start"] = s["start"].cpu().numpy()
        else:
            s["evec"] = torch.zeros(case["ned"] + 1, A.n, device=DEV, dtype=s["start"].dtype)
    else:
        Ls, diags = _batch_inputs(case, gen)
        s["batch"] = Batch.stencil5(Ls, diags)
        s["batch"].autotune(**_batch_options(case, seed))
        s["seed"] = seed
    return s


def _host(case):
    # A callback on device pointers goes with vectors on the device.
    return case["host"] and case["fmt"] != "callback"


def _batch_options(case, seed):
    return dict(ned=case["ned"], maxlan=case["maxlan"], tol=1e-8, restart=1, maxmv=100000, seed=1 + int(seed))


def run(s):
    case = s["case"]
    if case["kind"] == "solve":
        r = solve(s["op"], ned=case["ned"], maxlan=case["maxlan"], lohi=-1, tol=1e-8, restart=1,
                  maxmv=_maxmv(case), start=s["start"], basis_bits=case["bits"], device=not _host(case),
                  evec=s.get("evec"))
        # The converged pairs (the rest of the arrays cleared), or the
        # approximations of all wanted ones.
        k = r.nec or case["ned"]
        r.eval[k:] = 0.0
        r.evec[k:] = 0.0
        return {"eval": r.eval, "evec": _signed(r.evec, k, case["bits"])}
    # The eigenvalues; the residual estimates and counters of a converged
    # solve are diagnostics that depend on the last bits of the sums.
    return {"eval": s["batch"].solve(**_batch_options(case, s["seed"])).eval}


def _signed(v, k, bits):
    """The first k vectors with their free sign (phase) fixed by the largest
    entry, as a program does that stores or compares them; from a 32-bit
    basis, in the precision that they have."""
    if isinstance(v, np.ndarray):
        top = np.take_along_axis(v[:k], np.abs(v[:k]).argmax(axis=1)[:, None], axis=1)
        v[:k] *= np.conj(top) / np.abs(top)
        return v.astype(np.complex64 if np.iscomplexobj(v) else np.float32) if bits == 32 else v
    top = torch.gather(v[:k], 1, v[:k].abs().argmax(dim=1, keepdim=True))
    v[:k].mul_(top.conj() / top.abs())
    return v.to(torch.complex64 if v.is_complex() else torch.float32) if bits == 32 else v


def _maxmv(case):
    """Operator applications of `cycles` restart cycles: a full basis, then
    half-full ones (a restart of scheme 1 keeps about half)."""
    return case["maxlan"] + (case["cycles"] - 1) * ((case["maxlan"] - case["ned"]) // 2)


# ---- what a pass cannot do without ------------------------------------------
def work(case):
    if case["kind"] == "solve":
        cplx = case["family"] == "peierls"
        n = case["L"] ** 3 if case["family"] == "anderson" else case["L"] ** 2
        cs = 16 if cplx else 8
        sv = cs // 2 if case["bits"] == 32 else cs
        per_row = {"anderson": 7, "peierls": 5}.get(case["family"], 5)
        ned, maxlan = case["ned"], case["maxlan"]
        sizes = list(range(1, maxlan + 1))
        first = maxlan - (maxlan - ned) // 2
        while len(sizes) < _maxmv(case):
            sizes += list(range(first + 1, maxlan + 1))
        sizes = sizes[:_maxmv(case)]
        steps = len(sizes)
        # Every step applies the operator (its entries, x, y), reads the
        # basis to orthogonalise against it and writes one new vector; every
        # restart and the end read the basis and write the kept vectors.
        b = steps * n * (per_row * (cs + 4) + 2 * cs + sv) + sum(sizes) * n * sv
        b += case["cycles"] * n * sv * maxlan + (case["cycles"] - 1) * n * sv * first + n * cs * (ned + 1)
        mul = 8 if cplx else 2
        f = mul * n * (steps * per_row + 2.0 * sum(sizes)) + (mul / 2) * 2 * n * maxlan * (ned + (case["cycles"] - 1) * first)
        return {"bytes": float(b), "flops": float(f)}
    # Operator applications grow with L (475 on average at L = 152); the
    # basis is three quarters full on average.
    mid = 0.5 * (case["lo"] + case["hi"])
    rows = case["problems"] * (mid * mid + (case["hi"] - case["lo"]) ** 2 / 12.0)
    steps = 2.6 * mid + 80.0
    m = 0.75 * case["maxlan"]
    return {"bytes": rows * steps * 8.0 * (m + 3.0), "flops": rows * steps * (4.0 * m + 12.0)}


# ---- 64-bit values ------------------------------------------------------------
def _apply(n, cols, vals, inside):
    """x -> A x from padded rows (entries outside the grid are zero)."""
    if inside is not None:
        vals = torch.where(inside, vals, torch.zeros_like(vals))
        cols = torch.where(inside, cols, torch.zeros_like(cols))

    def f(x):
        y = vals[:, 0] * x[cols[:, 0]]
        for k in range(1, cols.shape[1]):
            y += vals[:, k] * x[cols[:, k]]
        return y
    return f


def _lanczos_values(apply, q, steps):
    """Ritz values (ascending) and residual norms of a `steps`-dimensional Krylov space, every
    vector orthogonalised twice against all before it."""
    V = torch.zeros(steps, q.numel(), device=DEV, dtype=q.dtype)
    q = q / torch.linalg.vector_norm(q)
    a, b = [], []
    for j in range(steps):
        V[j] = q
        r = apply(q)
        a.append(torch.vdot(q, r).real)
        for _ in range(2):
            r = r - torch.mv(V[:j + 1].transpose(0, 1), torch.mv(V[:j + 1].conj(), r))
        b.append(torch.linalg.vector_norm(r))
        q = r / b[-1]
    T = torch.diag(torch.stack(a)) + torch.diag(torch.stack(b[:-1]), 1) + torch.diag(torch.stack(b[:-1]), -1)
    w, z = torch.linalg.eigh(T.cpu())
    return w.numpy(), (b[-1].cpu() * z[-1].abs()).numpy()


def exact(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    if case["kind"] == "solve":
        # One cycle: the Ritz values of its Krylov space; none where some may
        # have converged, so that only those come back.  After restarts they
        # depend on the restart scheme's choices; the vectors are only
        # determined up to sign.
        if case["cycles"] != 1:
            return None
        n, cols, vals, inside = _entries(case, gen)
        q = _start(gen, n, vals.is_complex())
        ev, res = _lanczos_values(_apply(n, cols, vals, inside), q, case["maxlan"])
        if res[:case["ned"]].min() < 1e-6 * abs(ev).max():
            return None
        return {"eval": np.append(ev[:case["ned"]], 0.0), "evec": None}
    if case["problems"] > 64 or case["hi"] > 96:
        return None
    Ls, diags = _batch_inputs(case, gen)
    out = np.zeros((case["problems"], case["ned"]))
    for p, (L, d) in enumerate(zip(Ls, diags)):
        L = int(L)
        i = torch.arange(L * L, device=DEV)
        ix, iy = i % L, i // L
        cols = torch.stack([i, i - 1, i + 1, i - L, i + L], dim=1)
        vals = torch.full((L * L, 5), -1.0, device=DEV, dtype=torch.float64)
        vals[:, 0] = 4.0 + torch.as_tensor(d, device=DEV)
        inside = torch.stack([ix >= 0, ix > 0, ix < L - 1, iy > 0, iy < L - 1], dim=1)
        if L <= 32:
            A = torch.zeros(L * L, L * L, device=DEV, dtype=torch.float64)
            for k in range(5):
                m = inside[:, k]
                A[i[m], cols[m, k]] = vals[m, k]
            out[p] = torch.linalg.eigvalsh(A)[:case["ned"]].cpu().numpy()
        else:
            q = _rand(gen, L * L) - 0.5
            out[p] = _lanczos_values(_apply(L * L, cols, vals, inside), q, 320 + L)[0][:case["ned"]]
    return {"eval": out}
