"""CG that breaks down right at a periodic true-residual check: the scalar step
that finds rho = 0 follows the check, in the same iteration."""
import numpy as np
import pytest
import torch

import ainv
import oracle as O

pytestmark = pytest.mark.gpu


def test_rho_zero_at_a_periodic_check():
    """M is far too large for A (about 2^100 A^-1), so that r.z falls below the
    smallest number while p.q does not: alpha is then 0, and the next iteration
    finds the rho of the one before it 0.  The size of b sets the iteration;
    the oracle, which checks nothing, says which sizes meet the checks after 50
    and 100 iterations.  Every number is a double either way (the factors are
    powers of two), so iterates are the oracle's bits."""
    n = 300
    irp = np.concatenate([[0], np.cumsum(np.r_[2, np.full(n - 2, 3), 2])]).astype(np.int32)
    rows = np.repeat(np.arange(n), np.diff(irp))
    ja = (rows + np.concatenate([[0, 1], np.tile([-1, 0, 1], n - 2), [-1, 0]])).astype(np.int32)
    csr = irp, ja, np.where(ja == rows, 2.001, -1.0) * 2.0 ** 200
    one = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n)
    d = np.full(n, 2.0 ** -101)
    a, of = O.CSR(n, *csr), O.Factors(O.CSR(n, *one), O.CSR(n, *one), d)
    A, f = ainv.DeviceOperator(*csr), ainv.DeviceFactors(one, one, d, prec="FP32_ACC64")
    b = np.random.default_rng(1).uniform(-1, 1, n)
    met = set()
    for k in np.linspace(-488, -480, 400):
        bk = b * 2.0 ** k
        xr, it, _, rc = O.solve("CG", a, of, bk, eps=1e-300, itmax=400)
        if rc not in (-1, -3) or it - 1 not in (50, 100):  # it counts the one that broke down
            continue
        met.add(it - 1)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        res = A.solve(torch.from_numpy(bk).cuda(), x, f, "CG", 1e-300, 400)
        assert (res.info, res.iter, res.replacements) == (4102, it - 1, 0)
        assert np.array_equal(x.cpu().numpy(), xr)
    assert met == {50, 100}
