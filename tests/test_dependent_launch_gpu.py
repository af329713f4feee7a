"""Calls queued back to back, each on what the one before it wrote, against the
same calls with the device idle in between: kernels of several calls are
resident together then, and the shared intermediate is rewritten by each."""
import numpy as np
import pytest
import torch

import ainv
from util import build_factors, build_inverse_factors, device_factors

pytestmark = pytest.mark.gpu


def chain(f, x0, steps, wait, updates=False):
    x, y = x0.clone(), torch.zeros_like(x0)
    out = []
    for k in range(steps):
        f.apply(x, y, 3.0, 0.25 if k % 3 else 0.0, "NT"[k % 2])
        if wait:
            torch.cuda.synchronize()
        if updates and k % 5 == 4:
            f.update_a(x0.abs() + 1.0)
        if wait:
            torch.cuda.synchronize()
        x, y = y, x
        if k % 16 == 0:
            out.append(x.clone())
    torch.cuda.synchronize()
    return out + [x, y]


@pytest.mark.parametrize("updates", [False, True])
@pytest.mark.parametrize("idim,pattern,prec", [
    (12, "ainv", "FP64"), (40, "ainv", "FP32"),  # one launch per apply
    (54, "ainv", "FP64"), (58, "ainv", "BF16"), (66, "ainv", "FP32_ACC64"),
    (14, "invk", "FP64"), (24, "invk", "FP32"), (31, "invk", "BF16_ACC64"),
])
def test_chained_applies(idim, pattern, prec, updates):
    csr = ainv.pde.gen_pde3d(idim, "convdiff", (3.0, 2.0, -1.0))
    fac = build_factors(*csr) if pattern == "ainv" else build_inverse_factors("INVK", *csr)
    x0 = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, idim ** 3)).cuda()
    alone = chain(device_factors(fac, prec), x0, 97, True, updates)
    f = device_factors(fac, prec)
    for a, b in zip(alone, chain(f, x0, 97, False, updates)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("method", ["CG", "BICGSTAB"])
@pytest.mark.parametrize("prec", ["FP64", "FP32"])
def test_plain_loop_repeats(method, prec):
    """A solve without a preconditioner and one past the persistent loop's size,
    again on the same workspace with other systems in between."""
    n = 500_000
    irp = np.concatenate([[0], np.cumsum(np.r_[2, np.full(n - 2, 3), 2])]).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(irp))
    ja = (rows + np.concatenate([[0, 1], np.tile([-1, 0, 1], n - 2), [-1, 0]])).astype(np.int32)
    val = np.where(ja == rows, 2.5, -1.0)
    A = ainv.DeviceOperator(irp, ja, val)
    f = device_factors(build_factors(irp, ja, val), prec)
    bs = [torch.from_numpy(np.random.default_rng(k).uniform(-1, 1, n)).cuda() for k in range(2)]
    xs = {}
    for _ in range(3):
        for k, b in enumerate(bs):
            for pre in (f, None):
                x = torch.zeros_like(b)
                res = A.solve(b, x, pre, method, 1e-9, 300)
                assert res.converged
                r = b - torch.zeros_like(b)
                A.spmv(x, r, -1.0, 1.0)
                assert torch.linalg.norm(r) <= 1.05e-9 * torch.linalg.norm(b)
                want = xs.setdefault((k, pre is None), x)
                assert torch.equal(x, want)
