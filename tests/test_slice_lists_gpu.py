"""Sweeps and A products whose slices share offset lists, have their own, or
store a column per entry, with slice widths at the edges of a kernel step
(4 and 8 slots) and of a pack, and row counts around a slice: the device
results against the oracle's."""
import numpy as np
import pytest
import torch

import ainv
import oracle as O
from util import build_factors, device_factors, oracle_factors, relerr

pytestmark = pytest.mark.gpu


def triangle(n, widths, seed, upper, scattered_every):
    """Unit triangular CSR whose 32-row slice s has widths[s % len] entries per
    row at most: a band of fixed offsets, or random columns in every
    scattered_every-th slice; some entries missing."""
    rng = np.random.default_rng(seed)
    irp, ja, val = [0], [], []
    for r in range(n):
        s = r // 32
        w = widths[s % len(widths)]
        reach = n - 1 - r if upper else r
        if scattered_every and s % scattered_every == 0:
            k = min(w - 1, reach)
            off = rng.choice(np.arange(1, reach + 1), k, replace=False) if k else []
        else:
            off = [o for o in range(1, w) if o <= reach and rng.random() < 0.9]
        cols = sorted([r + o if upper else r - o for o in off] + [r])
        ja += cols
        val += [1.0 if c == r else rng.uniform(-0.4, 0.4) for c in cols]
        irp.append(len(ja))
    return np.array(irp, np.int32), np.array(ja, np.int32), np.array(val)


@pytest.mark.parametrize("prec", ["FP64", "FP32", "BF16", "FP32_ACC64", "BF16_ACC64"])
@pytest.mark.parametrize("n,widths,scattered", [
    (1, (1,), 0), (31, (2,), 0), (33, (4,), 0), (1000, (4, 3, 1), 0), (1000, (5,), 0),
    (2000, (8, 9), 0), (2000, (4, 70), 0), (4097, (3, 5, 8), 2), (4100, (7,), 1),
])
def test_mixed_slices(prec, n, widths, scattered):
    wt = triangle(n, widths, 1, False, scattered)
    z = triangle(n, widths, 2, True, scattered)
    rng = np.random.default_rng(3)
    d, x, y0 = rng.uniform(0.5, 2.0, n), rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    f = ainv.DeviceFactors(wt, z, d, prec=prec)

    def rnd(v):
        if prec.startswith("FP32"):
            return v.astype(np.float32).astype(np.float64)
        if prec.startswith("BF16"):
            return torch.from_numpy(v).float().bfloat16().double().numpy()
        return v

    of = O.Factors(O.CSR(n, wt[0], wt[1], rnd(wt[2])), O.CSR(n, z[0], z[1], rnd(z[2])), rnd(d))
    for trans, beta in (("N", 0.0), ("N", -0.5), ("T", 0.25)):
        xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y0).cuda()
        f.apply(xd, yd, 1.5, beta, trans)
        got = yd.cpu().numpy()
        ref = O.ainv_apply(of, x, 1.5, beta, y0, trans)
        if prec in ("FP32", "BF16"):
            # FP32 sums of at most 71 products of size < 1 in two sweeps, and t
            # rounded to FP32 between them
            tol = 2 * 71 * 2.0 ** -24 * 4
        else:
            # the same roundings in the same order; 'T' sums the oracle's
            # products by columns instead of rows
            tol = 0.0 if trans == "N" else 1e-13
        assert relerr(got, ref) <= tol, (prec, trans, beta)


@pytest.mark.parametrize("n,widths,scattered", [(31, (3,), 0), (1000, (4, 9), 0), (4097, (5,), 2)])
def test_mixed_slices_product(n, widths, scattered):
    a = triangle(n, widths, 5, True, scattered)
    x = np.random.default_rng(6).uniform(-1, 1, n)
    A = ainv.DeviceOperator(*a)
    xd, yd = torch.from_numpy(x).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
    A.spmv(xd, yd, 1.0, 0.0)
    assert np.array_equal(yd.cpu().numpy(), O.spmv(O.CSR(n, *a), x))


@pytest.mark.parametrize("scattered", [0, 1])
def test_zero_slots_do_not_read(scattered):
    """An infinite element of x reaches only the rows that hold its column:
    missing entries of a slice's shared list add nothing."""
    n = 200
    wt, z = triangle(n, (5,), 7, False, scattered), triangle(n, (5,), 8, True, scattered)
    x = np.random.default_rng(9).uniform(-1, 1, n)
    x[77] = np.inf
    f = ainv.DeviceFactors(wt, z, np.ones(n))
    yd = torch.zeros(n, dtype=torch.float64, device="cuda")
    f.apply(torch.from_numpy(x).cuda(), yd)
    of = O.Factors(O.CSR(n, *wt), O.CSR(n, *z), np.ones(n))
    assert np.array_equal(yd.cpu().numpy(), O.ainv_apply(of, x), equal_nan=True)


@pytest.mark.parametrize("idim", [24, 40, 53, 54])
def test_one_launch_apply(idim):
    """Grids on both sides of the largest apply that goes out as one launch:
    the intermediate is left as the sweeps leave it, x and y may be the same
    vector, and a captured apply can be replayed on new contents."""
    rng = np.random.default_rng(2)
    csr = ainv.pde.gen_pde3d(idim, "convdiff", (3.0, 2.0, -1.0))
    f = build_factors(*csr)
    n = len(f["d"])
    df, of = device_factors(f), oracle_factors(f)
    x1, x2 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    for trans in "NT":
        x, y = torch.from_numpy(x1).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
        df.apply(x, y, 1.0, 0.0, trans)
        first = y.clone()
        assert relerr(first.cpu().numpy(), O.ainv_apply(of, x1, 1.0, 0.0, x1, trans)) <= (
            0.0 if trans == "N" else 1e-13)
        df.apply_stage(2, y=y, alpha=2.0, trans=trans)
        assert torch.equal(y, 2.0 * first)
        both = x.clone()
        df.apply(both, both, 1.0, 0.0, trans)
        assert torch.equal(both, first)
        part = torch.cat([x, x])
        df.apply(part[:n], part[n // 2:n // 2 + n], 1.0, 0.0, trans)
        assert torch.equal(part[n // 2:n // 2 + n], first)
    x, y = torch.from_numpy(x1).cuda(), torch.zeros(n, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        df.apply(x, y, stream=torch.cuda.current_stream())
        df.apply(y, x, stream=torch.cuda.current_stream())
    for v in (x1, x2):
        x.copy_(torch.from_numpy(v))
        g.replay()
        torch.cuda.synchronize()
        once = O.ainv_apply(of, v)
        assert np.array_equal(y.cpu().numpy(), once)
        assert np.array_equal(x.cpu().numpy(), O.ainv_apply(of, once))


def test_applies_after_update_a():
    """An apply right behind update_a reads the new diagonal."""
    csr = ainv.pde.gen_pde3d(24, "poisson")
    f = build_factors(*csr)
    n = len(f["d"])
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    a, b = device_factors(f), device_factors(f)
    ya, yb = torch.zeros_like(x), torch.zeros_like(x)
    a.update_a(x)
    torch.cuda.synchronize()
    a.apply(x, ya)
    b.apply(x, yb)
    b.update_a(x)
    b.apply(x, yb)
    assert torch.equal(ya, yb)
