"""Waits of the persistent loop that run out (limit 0: the first block that has
to wait gives up): a loop that any block left is reported as timed out, one
that none left is right, and the next one on the same objects is right."""
import numpy as np
import pytest
import torch

import ainv
from util import build_factors, device_factors

pytestmark = pytest.mark.gpu
TIMEOUT = 4106


def system(idim, kind="poisson", prec="FP64"):
    csr = ainv.pde.gen_pde3d(idim, kind, (4.0, -3.0, 2.0))
    b = np.random.default_rng(1).uniform(-1, 1, idim ** 3)
    return ainv.DeviceOperator(*csr), device_factors(build_factors(*csr), prec), b


@pytest.mark.parametrize("method,idim", [("CG", 10), ("BICGSTAB", 10), ("CG", 40),
                                         ("BICGSTAB", 40), ("CG", 60)])
@pytest.mark.parametrize("itmax", [0, 1, 200])
def test_solve(monkeypatch, method, idim, itmax):
    A, f, b = system(idim)
    bd = torch.from_numpy(b).cuda()
    ref = torch.zeros_like(bd)
    want = A.solve(bd, ref, f, method, 1e-9, itmax)
    gave_up = 0
    for _ in range(100):
        monkeypatch.setenv("AINV_WAIT_MS", "0")
        x = torch.zeros_like(bd)
        try:
            got = A.solve(bd, x, f, method, 1e-9, itmax)
        except ainv.AinvError as e:
            assert e.info == TIMEOUT, e
            gave_up += 1
        else:
            assert (got.info, got.iter) == (want.info, want.iter) and torch.equal(x, ref)
        monkeypatch.delenv("AINV_WAIT_MS")
    if itmax == 200 and idim >= 40:  # two blocks may arrive together every time, hundreds do not
        assert gave_up == 100
    x = torch.zeros_like(bd)
    got = A.solve(bd, x, f, method, 1e-9, itmax)
    assert (got.info, got.iter, got.err) == (want.info, want.iter, want.err)
    assert torch.equal(x, ref)


def test_block_zero_passes_alone(monkeypatch):
    """Block 0 has a group more than the others, so it is the last at the only
    barrier of a solve of no iterations: it stores a finished state while every
    other block has given up."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (4 * sms + 2) * 256  # two blocks of two teams per SM, a group of 256 rows per team
    irp = np.concatenate([[0], np.cumsum(np.r_[2, np.full(n - 2, 3), 2])]).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(irp))
    ja = (rows + np.concatenate([[0, 1], np.tile([-1, 0, 1], n - 2), [-1, 0]])).astype(np.int32)
    csr = irp, ja, np.where(ja == rows, 2.5, -1.0)
    A, f = ainv.DeviceOperator(*csr), device_factors(build_factors(*csr))
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    assert A.solve(b, x, f, "CG", 1e-9, 0).info == 4104
    monkeypatch.setenv("AINV_WAIT_MS", "0")
    for _ in range(20):
        with pytest.raises(ainv.AinvError) as e:
            A.solve(b, x, f, "CG", 1e-9, 0)
        assert e.value.info == TIMEOUT
    monkeypatch.delenv("AINV_WAIT_MS")
    assert A.solve(b, x, f, "CG", 1e-9, 100).converged


def test_server(monkeypatch):
    cases = [system(20, "convdiff", "FP32"), system(30, "poisson", "FP32")]
    refs = []
    for a, f, b in cases:
        x = torch.zeros(len(b), dtype=torch.float64, device="cuda")
        assert a.solve(torch.from_numpy(b).cuda(), x, f, "BICGSTAB", 1e-9, 300).converged
        refs.append(x.cpu().numpy())
    for limit in ("0", None):
        if limit is None:
            monkeypatch.delenv("AINV_WAIT_MS")
        else:
            monkeypatch.setenv("AINV_WAIT_MS", limit)
        gave_up = 0
        with ainv.SolveServer(max_slots=3, hbm_bytes=1 << 28, iters_per_launch=2) as srv:
            ops = [srv.add_operator(a, f) for a, f, _ in cases]
            xs = [np.zeros(len(cases[q % 2][2])) for q in range(12)]
            ids = [srv.submit(ops[q % 2], cases[q % 2][2], x, 1e-9, 300)
                   for q, x in enumerate(xs)]
            for q, i in enumerate(ids):
                try:
                    res = srv.wait(i, timeout=60.0)
                except ainv.AinvError as e:
                    assert e.info == TIMEOUT and "time limit" in str(e), e
                    gave_up += 1
                else:
                    assert res.converged and np.array_equal(xs[q], refs[q % 2])
        assert gave_up == (0 if limit is None else 12)
