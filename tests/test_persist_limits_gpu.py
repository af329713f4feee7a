"""Which systems run in the persistent Krylov loop.  Its waits are the only ones
of a device solve, so with a limit of 0 a system that takes it times out, and
one that takes the plain loop is solved."""
import numpy as np
import pytest
import torch

import ainv
from util import build_factors, build_inverse_factors, device_factors

pytestmark = pytest.mark.gpu
TIMEOUT = 4106


def stencil27(m):
    """27-point operator: 27 on the diagonal, -1 for every neighbour."""
    g = np.arange(m ** 3).reshape(m, m, m)
    rows, cols = [], []
    for d in np.ndindex(3, 3, 3):
        off = [k - 1 for k in d]
        rows.append(g[tuple(slice(max(0, -k), m - max(0, k)) for k in off)].ravel())
        cols.append(g[tuple(slice(max(0, k), m - max(0, -k)) for k in off)].ravel())
    r, c = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    irp = np.zeros(m ** 3 + 1, np.int32)
    np.cumsum(np.bincount(r), out=irp[1:])
    return irp, c.astype(np.int32), np.where(r == c, 27.0, -1.0)


def tridiagonal(n):
    irp = np.concatenate([[0], np.cumsum(np.r_[2, np.full(n - 2, 3), 2])]).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(irp))
    ja = (rows + np.concatenate([[0, 1], np.tile([-1, 0, 1], n - 2), [-1, 0]])).astype(np.int32)
    return irp, ja, np.where(ja == rows, 2.05, -1.0)


def system(points, factors, idim, prec):
    """The factors have 11 slots per row for 3 points, 4 (AINV) or 23 (INVK) for
    7, and 1 or 131 for 27."""
    csr = (stencil27(idim) if points == 27 else tridiagonal(idim ** 3) if points == 3 else
           ainv.pde.gen_pde3d(idim, "poisson", (0., 0., 0.)))
    fac = build_factors(*csr) if factors == "AINV" else build_inverse_factors(factors, *csr)
    return ainv.DeviceOperator(*csr), device_factors(fac, prec)


@pytest.mark.parametrize("points,factors,idim,prec,persistent", [
    (7, "AINV", 70, "FP64", True), (7, "AINV", 70, "BF16_ACC64", True),
    (7, "INVK", 52, "FP64", True), (7, "INVK", 56, "FP64", False),
    (7, "INVK", 60, "FP32", True), (7, "INVK", 69, "FP32", False),
    (7, "INVK", 56, "BF16", False), (7, "INVK", 56, "BF16_ACC64", False),
    (27, "AINV", 60, "FP64", True), (27, "AINV", 70, "FP64", False),
    (27, "INVK", 20, "FP64", False), (27, "INVK", 20, "FP32_ACC64", False),
])
def test_solve(monkeypatch, points, factors, idim, prec, persistent):
    """The sizes lie on both sides of where the two loops' times cross."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 multiprocessors")
    A, f = system(points, factors, idim, prec)
    b = torch.from_numpy(np.random.default_rng(0).uniform(-1, 1, idim ** 3)).cuda()
    for method in ("CG", "BICGSTAB"):
        x = torch.zeros_like(b)
        want = A.solve(b, x, f, method, 1e-6, 60)
        monkeypatch.setenv("AINV_WAIT_MS", "0")
        y = torch.zeros_like(b)
        if persistent:
            with pytest.raises(ainv.AinvError) as e:
                A.solve(b, y, f, method, 1e-6, 60)
            assert e.value.info == TIMEOUT
        else:
            got = A.solve(b, y, f, method, 1e-6, 60)
            assert (got.info, got.iter, got.err) == (want.info, want.iter, want.err)
            assert torch.equal(x, y)
        monkeypatch.delenv("AINV_WAIT_MS")


@pytest.mark.parametrize("points,factors,idim,prec,persistent", [
    (7, "AINV", 24, "FP32", True), (7, "INVK", 40, "FP64", True),
    (7, "INVK", 50, "BF16_ACC64", True), (7, "INVK", 86, "BF16_ACC64", False),
    (3, "AINV", 80, "FP32_ACC64", True), (3, "AINV", 90, "FP32_ACC64", False),
    (27, "AINV", 50, "FP64", True), (27, "INVK", 20, "FP64", False),
])
def test_server(monkeypatch, points, factors, idim, prec, persistent):
    """One request, so that it is the whole mix."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 multiprocessors")
    A, f = system(points, factors, idim, prec)
    b = np.random.default_rng(0).uniform(-1, 1, idim ** 3)
    x = torch.zeros(idim ** 3, dtype=torch.float64, device="cuda")
    assert A.solve(torch.from_numpy(b).cuda(), x, f, "BICGSTAB", 1e-6, 200).converged
    y = np.zeros_like(b)
    monkeypatch.setenv("AINV_WAIT_MS", "0")
    with ainv.SolveServer(max_slots=2, hbm_bytes=1 << 30) as srv:
        i = srv.submit(srv.add_operator(A, f), b, y, 1e-6, 200)
        if persistent:
            with pytest.raises(ainv.AinvError) as e:
                srv.wait(i, timeout=60.0)
            assert e.value.info == TIMEOUT and "time limit" in str(e.value)
        else:
            assert srv.wait(i, timeout=60.0).converged
            assert np.array_equal(y, x.cpu().numpy())
