"""The persistent Krylov loop at the sizes where its split changes: one slice,
one group, a partly filled team, one and two blocks per SM, one and more
ranges of sums, the last size it takes and the first it does not; more
iterations than one launch runs; and the residual replacement.  Iterates
equal the oracle's (FP64) or the solve server's (reduced precision) bit for
bit."""
import numpy as np
import pytest
import torch

import ainv
import oracle as O
from util import build_factors, build_inverse_factors, device_factors, oracle_factors

pytestmark = pytest.mark.gpu


def band_operator(n, seed=0):
    """A diagonally dominant tridiagonal-plus-far-band operator of n rows."""
    rng = np.random.default_rng(seed)
    offs = sorted({0, 1, -1, 37, -37})
    rows = [(r, [r + o for o in offs if 0 <= r + o < n]) for r in range(n)]
    irp = np.zeros(n + 1, np.int32)
    ja, val = [], []
    for r, cols in rows:
        for c in cols:
            ja.append(c)
            val.append(4.5 if c == r else -1.0 + 0.2 * rng.random())
        irp[r + 1] = len(ja)
    return irp, np.array(ja, np.int32), np.array(val)


def check(method, csr, f, eps=1e-9, itmax=500):
    n = len(csr[0]) - 1
    b = np.random.default_rng(1).uniform(-1, 1, n)
    a = O.CSR(n, *csr)
    xr, it, err, rc, hist = O.solve(method, a, oracle_factors(f), b, eps=eps, itmax=itmax,
                                    history=True)
    A = ainv.DeviceOperator(*csr)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    res = A.solve(torch.from_numpy(b).cuda(), x, device_factors(f), method, eps, itmax)
    if rc == -3:  # the oracle counts the iteration that broke down, the device does not
        assert res.info == 4102 and res.iter == it - 1
        return res
    assert res.iter == it and (res.info == 0) == (rc == 0), (res, it, rc)
    np.testing.assert_array_equal(A.history()[:len(hist)], hist[:len(A.history())])
    np.testing.assert_array_equal(x.cpu().numpy(), xr)
    return res


@pytest.mark.parametrize("method", ["CG", "BICGSTAB"])
@pytest.mark.parametrize("n", [1, 31, 33, 256, 257, 1000, 4097])
def test_small(method, n):
    check(method, band_operator(n), build_factors(*band_operator(n)))


@pytest.mark.parametrize("method,idim", [("CG", 40), ("CG", 41), ("BICGSTAB", 42),
                                         ("BICGSTAB", 43), ("CG", 76), ("BICGSTAB", 77)])
def test_split(method, idim):
    kind = "poisson" if method == "CG" else "convdiff"
    csr = ainv.pde.gen_pde3d(idim, kind, (4.0, -3.0, 2.0))
    check(method, csr, build_factors(*csr))


@pytest.mark.parametrize("method,idim", [("CG", 17), ("BICGSTAB", 45)])
def test_wide_factors(method, idim):
    kind = "poisson" if method == "CG" else "convdiff"
    csr = ainv.pde.gen_pde3d(idim, kind, (4.0, -3.0, 2.0))
    check(method, csr, build_inverse_factors("INVK", *csr))


def test_several_launches():
    """2100 iterations without convergence: three launches of the loop."""
    csr = ainv.pde.gen_pde3d(24, "poisson")
    res = check("CG", csr, build_factors(*csr), eps=1e-300, itmax=2100)
    assert res.iter > 1024 or res.info != 0


@pytest.mark.parametrize("prec", ["FP32", "BF16"])
def test_replacement_equals_served(prec):
    """A tolerance below what the recurrence confirms: the residual is
    replaced by b - A x and the loop goes on, as in the server's kernels."""
    csr = ainv.pde.gen_pde3d(30, "convdiff", (9.0, -3.0, 2.0))
    n = len(csr[0]) - 1
    f, A = device_factors(build_factors(*csr), prec), ainv.DeviceOperator(*csr)
    b = np.random.default_rng(1).uniform(-1, 1, n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    res = A.solve(torch.from_numpy(b).cuda(), x, f, "BICGSTAB", 2e-16, 300)
    xs = np.zeros(n)
    with ainv.SolveServer(max_slots=1, hbm_bytes=1 << 28) as srv:
        got = srv.wait(srv.submit(srv.add_operator(A, f), b, xs, 2e-16, 300))
    assert res.verify_fails > 0 or res.replacements > 0
    assert (res.info, res.iter, res.err) == (got.status, got.iter, got.err)
    np.testing.assert_array_equal(x.cpu().numpy(), xs)


def test_solution_over_right_hand_side():
    """x and b may be the same vector: b is read before x is written."""
    csr = ainv.pde.gen_pde3d(20, "poisson")
    n = len(csr[0]) - 1
    f, A = device_factors(build_factors(*csr)), ainv.DeviceOperator(*csr)
    b = torch.rand(n, dtype=torch.float64, device="cuda")
    x = b.clone()
    A.solve(b.clone(), x, f, "CG", 1e-10, 200)
    both = b.clone()
    A.solve(both, both, f, "CG", 1e-10, 200)
    assert torch.equal(both, x)


def test_server_forms_follow_each_other():
    """Small requests (persistent loop), joined by large ones and by another
    precision (batched kernels), alone again at the end: every result is the
    single solve's.  Three iterations per launch, so p changes buffers."""
    cases = []
    for idim, prec, kind in [(20, "FP32", "convdiff"), (24, "FP32", "poisson"),
                             (96, "FP32", "convdiff"), (24, "FP64", "convdiff")]:
        csr = ainv.pde.gen_pde3d(idim, kind, (6.0, -3.0, 2.0))
        cases.append((ainv.DeviceOperator(*csr), device_factors(build_factors(*csr), prec), idim ** 3))
    order = [0, 1, 0, 1, 2, 0, 1, 3, 2, 2, 2, 1, 0, 3, 0, 1]
    bs = [np.random.default_rng(k).uniform(-1, 1, cases[c][2]) for k, c in enumerate(order)]
    xs = [np.zeros(cases[c][2]) for c in order]
    with ainv.SolveServer(max_slots=6, hbm_bytes=1 << 30, iters_per_launch=3) as srv:
        ops = [srv.add_operator(a, f) for a, f, _ in cases]
        ids = [srv.submit(ops[c], b, x, 1e-9, 400) for c, b, x in zip(order, bs, xs)]
        got = [srv.wait(i) for i in ids]
    for c, b, x, g in zip(order, bs, xs, got):
        a, f, n = cases[c]
        ref = torch.zeros(n, dtype=torch.float64, device="cuda")
        res = a.solve(torch.from_numpy(b).cuda(), ref, f, "BICGSTAB", 1e-9, 400)
        assert (g.status, g.iter, g.err) == (res.info, res.iter, res.err)
        np.testing.assert_array_equal(x, ref.cpu().numpy())


@pytest.mark.parametrize("method,idim", [("CG", 84), ("BICGSTAB", 84), ("BICGSTAB", 85)])
def test_largest(method, idim):
    """The largest grid of the persistent loop, and the first of the plain one."""
    kind = "poisson" if method == "CG" else "convdiff"
    csr = ainv.pde.gen_pde3d(idim, kind, (4.0, -3.0, 2.0))
    check(method, csr, build_factors(*csr))


@pytest.mark.parametrize("method", ["CG", "BICGSTAB"])
@pytest.mark.parametrize("offs", [(-1, 0, 1), (-40, -1, 0, 1, 40, 41), (-3, 0, 1, 7)])
def test_other_packs(method, offs):
    """Operators and factors whose layout packs differ from those with kernels
    of their own (slices of 2, 3, 4 and 6 slots)."""
    rng = np.random.default_rng(4)
    n = 5000
    irp, ja, val = [0], [], []
    for r in range(n):
        cols = [r + o for o in offs if 0 <= r + o < n]
        ja += cols
        val += [8.0 if c == r else -1.0 + 0.1 * rng.random() for c in cols]
        irp.append(len(ja))
    csr = np.array(irp, np.int32), np.array(ja, np.int32), np.array(val)
    check(method, csr, build_factors(*csr))
