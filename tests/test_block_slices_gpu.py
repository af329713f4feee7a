"""Multi-right-hand-side CG on slices that its kernels treat apart: wider than
the slots kept in registers (INVK factors), a column for every entry, one slot,
and rows that do not fill a slice."""
import numpy as np
import pytest
import torch

import ainv
import oracle as O
from util import build_factors, build_inverse_factors, device_factors, within_spread

pytestmark = pytest.mark.gpu


def spd_scattered(n, per_row, seed):
    """Symmetric, diagonally dominant, random columns."""
    rng = np.random.default_rng(seed)
    d = np.zeros((n, n))
    for r in range(n):
        for c in rng.choice(n, per_row, replace=False):
            if c != r:
                d[r, c] = d[c, r] = -rng.random()
    d[np.arange(n), np.arange(n)] = 1.0 - d.sum(axis=1)
    irp = np.concatenate([[0], np.cumsum((d != 0).sum(axis=1))]).astype(np.int32)
    ja = np.nonzero(d)[1].astype(np.int32)
    return irp, ja, d[d != 0]


@pytest.mark.parametrize("prec", ["FP64", "FP32", "BF16_ACC64"])
@pytest.mark.parametrize("case", ["invk", "scattered", "diagonal"])
def test_columns_solve_as_alone(prec, case):
    if case == "invk":
        csr = ainv.pde.gen_pde3d(17, "poisson")
        f = build_inverse_factors("INVK", *csr)
    elif case == "scattered":
        csr = spd_scattered(700, 6, 3)
        f = build_factors(*csr)
    else:
        csr = (np.arange(46, dtype=np.int32), np.arange(45, dtype=np.int32),
               np.linspace(1.0, 3.0, 45))
        f = build_factors(*csr)
    n, m = len(csr[0]) - 1, 5
    b = np.random.default_rng(1).uniform(-1, 1, (n, m))
    A, df = ainv.DeviceOperator(*csr), device_factors(f, prec)
    B = torch.from_numpy(b).cuda()
    X = torch.zeros_like(B)
    res = A.block_solve(B, X, df, 1e-9, 400)
    assert res.converged
    a = O.CSR(n, *csr)
    for k in range(m):
        x = X[:, k].cpu().numpy()
        assert np.linalg.norm(b[:, k] - O.spmv(a, x)) <= 1.05e-9 * np.linalg.norm(b[:, k])
        one = torch.zeros(n, dtype=torch.float64, device="cuda")
        it = A.solve(B[:, k].contiguous(), one, df, "CG", 1e-9, 400).iter
        assert within_spread(res.iters[k], it, it)
