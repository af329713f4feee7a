"""Performance cases: what a user of the framework has it do, with sizes.

Every case goes through the public Python entry points.  There are four
kinds of call:

  apply  DeviceFactors.apply, y = alpha * op(M) x + beta * y, M = Z D^-1 W^T
         (the preconditioner inside somebody else's Krylov loop);
  solve  DeviceOperator.solve, preconditioned CG / BiCGSTAB with istop=2;
  block  DeviceOperator.block_solve, CG on up to 32 right-hand sides;
  serve  SolveServer, several requests on several operators in flight.

Operators are the 7-point operators of `ainv.pde` on an idim^3 grid.  The
factors of the solves come from the library's own AINV build (drop 0.1, cap
20).  Those of the applies have the patterns that the builds give on these
operators ("ainv": 4 entries per row; "invk": the 23 of INVK(1,1);
"scattered": 4 entries per row whose columns share no pattern, as a general
unstructured matrix has) with values drawn from the seed in the builds' range,
so no two rows repeat.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "mld-ainv_b200"))
import ainv  # noqa: E402

PRECS = ("FP64", "FP32", "BF16", "FP32_ACC64", "BF16_ACC64")
VALUE_BYTES = {"FP64": 8, "FP32": 4, "BF16": 2, "FP32_ACC64": 4, "BF16_ACC64": 2}

# (dz, dy, dx) of a row of W^T; Z has the mirrored list.
AINV_STENCIL = [(-1, 0, 0), (0, -1, 0), (0, 0, -1)]
INVK_STENCIL = [(-2, 0, 0), (-2, 0, 1), (-2, 0, 2), (-2, 1, 0), (-2, 1, 1), (-2, 2, 0),
                (-1, -1, 0), (-1, -1, 1), (-1, -1, 2), (-1, 0, -1), (-1, 0, 0), (-1, 0, 1),
                (-1, 1, -1), (-1, 1, 0), (0, -2, 0), (0, -2, 1), (0, -2, 2), (0, -1, -1),
                (0, -1, 0), (0, -1, 1), (0, 0, -2), (0, 0, -1)]


def listed():
    return [
        # the smallest grid of the serving mix: two launches and their latency
        dict(name="apply_24", kind="apply", pattern="ainv", idim=24, prec="FP64", trans="N",
             alpha=1.0, beta=0.0),
        # the small Poisson configuration
        dict(name="apply_40", kind="apply", pattern="ainv", idim=40, prec="FP64", trans="N",
             alpha=1.0, beta=0.0),
        # the transposed apply added to y, rows not a multiple of a slice
        dict(name="apply_97_T", kind="apply", pattern="ainv", idim=97, prec="FP64", trans="T",
             alpha=-1.0, beta=0.5),
        # the headline apply: factors well past the L2
        dict(name="apply_200", kind="apply", pattern="ainv", idim=200, prec="FP64", trans="N",
             alpha=1.0, beta=0.0),
        # reduced-precision factors, FP32 and BF16 accumulated in FP32
        dict(name="apply_128_fp32", kind="apply", pattern="ainv", idim=128, prec="FP32",
             trans="N", alpha=1.0, beta=0.0),
        dict(name="apply_101_bf16", kind="apply", pattern="ainv", idim=101, prec="BF16",
             trans="N", alpha=1.0, beta=0.0),
        # the denser INVK(1,1) factors
        dict(name="apply_64_invk", kind="apply", pattern="invk", idim=64, prec="FP64", trans="N",
             alpha=1.0, beta=0.0),
        # a general sparsity pattern: a column for every entry
        dict(name="apply_90_scattered", kind="apply", pattern="scattered", idim=90, prec="FP64",
             trans="N", alpha=1.0, beta=0.0),
        # one small system solved at once: latency of the Krylov loop
        dict(name="solve_40_cg", kind="solve", operator="poisson", idim=40, method="CG",
             prec="FP64", eps=1e-9),
        # a mid-size nonsymmetric system
        dict(name="solve_100_bicgstab", kind="solve", operator="convdiff", idim=100,
             method="BICGSTAB", prec="FP64", eps=1e-9),
        # 32 right-hand sides together, single-precision factors
        dict(name="block_64_32rhs", kind="block", operator="poisson", idim=64, rhs=32,
             prec="FP32", eps=1e-9),
        # the serving mix: requests on operators of two sizes in flight
        dict(name="serve_8_requests", kind="serve", idim=31, idim2=48, requests=8, prec="FP32",
             eps=1e-8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("apply", "apply", "apply", "apply", "solve", "solve", "block", "serve"))
    if kind == "apply":
        pattern = rng.choice(("ainv", "ainv", "ainv", "invk", "scattered"))
        hi = {"ainv": 140, "invk": 64, "scattered": 96}[pattern]
        return dict(kind=kind, pattern=pattern, idim=_log_int(rng, 20, hi),
                    prec=rng.choice(("FP64", "FP64") + PRECS), trans=rng.choice("NNT"),
                    alpha=rng.choice((1.0, -1.0, round(rng.uniform(0.1, 2.0), 3))),
                    beta=rng.choice((0.0, 0.0, round(rng.uniform(-0.9, 0.9), 3))))
    if kind == "solve":
        method = rng.choice(("CG", "BICGSTAB"))
        return dict(kind=kind, operator="poisson" if method == "CG" else "convdiff",
                    idim=_log_int(rng, 20, 96), method=method,
                    prec=rng.choice(("FP64", "FP64", "FP32_ACC64", "BF16_ACC64")), eps=1e-9)
    if kind == "block":
        return dict(kind=kind, operator="poisson", idim=_log_int(rng, 20, 60),
                    rhs=rng.randint(2, 32), prec=rng.choice(("FP64", "FP32", "FP32_ACC64")),
                    eps=1e-9)
    return dict(kind=kind, idim=_log_int(rng, 24, 40), idim2=_log_int(rng, 24, 56),
                requests=rng.randint(2, 16), prec=rng.choice(("FP64", "FP32")), eps=1e-8)


# ---------------------------------------------------------------- inputs --
def _stencil_csr(m, stencil, rng, mirror):
    """CSR of a unit triangular factor with the neighbours of `stencil`
    (mirrored for Z), off-diagonal magnitudes falling with the distance."""
    n = m ** 3
    sg = -1 if mirror else 1
    entries = [(sg * (dz * m * m + dy * m + dx), (sg * dz, sg * dy, sg * dx))
               for dz, dy, dx in stencil] + [(0, (0, 0, 0))]
    entries.sort()
    valid = np.zeros((m, m, m, len(entries)), bool)
    vals = rng.random((m, m, m, len(entries)))
    cols = np.arange(n, dtype=np.int32).reshape(m, m, m, 1) + \
        np.array([e[0] for e in entries], np.int32)
    for k, (off, d) in enumerate(entries):
        box = tuple(slice(max(0, -c), m - max(0, c)) for c in d)
        valid[box + (k,)] = True
        if off == 0:
            vals[..., k] = 1.0
        else:
            dist = sum(abs(c) for c in d)
            vals[..., k] = (0.17 + 0.04 * vals[..., k]) * 0.3 ** (dist - 1)
    irp = np.zeros(n + 1, np.int32)
    np.cumsum(valid.sum(axis=-1, dtype=np.int32).reshape(-1), out=irp[1:])
    return irp, cols[valid], vals[valid]


def _scattered_csr(m, rng, mirror):
    """A unit triangular factor with three off-diagonal entries per row at
    random columns within m^2 of the diagonal, fewer where those leave the matrix."""
    n, third = m ** 3, max(1, m * m // 3)
    dist = rng.integers(1, third + 1, (n, 3), dtype=np.int32) + \
        np.array([2 * third, third, 0], np.int32)
    rows = np.arange(n, dtype=np.int32)[:, None]
    cols = np.concatenate([rows - dist, rows], axis=1)
    vals = 0.17 + 0.04 * rng.random((n, 4))
    vals[:, 3] = 1.0
    if mirror:
        cols = np.concatenate([rows, rows + dist[:, ::-1]], axis=1)
        vals = np.ascontiguousarray(vals[:, ::-1])
    valid = (cols >= 0) & (cols < n)
    irp = np.zeros(n + 1, np.int32)
    np.cumsum(valid.sum(axis=1, dtype=np.int32), out=irp[1:])
    return irp, cols[valid], vals[valid]


def _apply_inputs(case, seed):
    m = case["idim"]
    rng = np.random.default_rng(seed)
    if case["pattern"] == "scattered":
        wt, z = _scattered_csr(m, rng, False), _scattered_csr(m, rng, True)
    else:
        stencil = AINV_STENCIL if case["pattern"] == "ainv" else INVK_STENCIL
        wt, z = _stencil_csr(m, stencil, rng, False), _stencil_csr(m, stencil, rng, True)
    n = m ** 3
    return wt, z, 0.1 + 0.2 * rng.random(n), rng.uniform(-1.0, 1.0, n), rng.uniform(-1.0, 1.0, n)


def _operator(kind, m):
    return ainv.pde.gen_pde3d(m, kind, (10 / np.sqrt(3),) * 3)


def _csr_times(csr, x):
    irp, ja, val = csr
    return np.add.reduceat((val * x.T[..., ja]), irp[:-1], axis=-1).T


def _factors(csr, prec):
    sv = ainv.mld_d_ainv_solver_type()
    sv.cseti("SUB_FILLIN", 20)
    sv.csetr("SUB_ILUTHRS", 0.1)
    if sv.build(*csr, amold=prec) != 0:
        raise RuntimeError(ainv.last_error())
    return sv


def _solution(case, seed):
    """The solution that a solve of this case is to find."""
    rng = np.random.default_rng(seed)
    n = case["idim"] ** 3
    if case["kind"] == "block":
        return rng.uniform(-1.0, 1.0, (n, case["rhs"]))
    if case["kind"] == "serve":
        return [rng.uniform(-1.0, 1.0, case["idim2" if q % 2 else "idim"] ** 3)
                for q in range(case["requests"])]
    return rng.uniform(-1.0, 1.0, n)


def prepare(case, seed):
    if case["kind"] == "apply":
        wt, z, d, x, y = _apply_inputs(case, seed)
        f = ainv.DeviceFactors(wt, z, d, prec=case["prec"])
        return dict(case=case, f=f, x=torch.from_numpy(x).cuda(), y=torch.from_numpy(y).cuda())
    if case["kind"] == "serve":
        ops = []
        srv = ainv.SolveServer(max_slots=16, hbm_bytes=1 << 30)
        for kind, m in (("convdiff", case["idim"]), ("poisson", case["idim2"])):
            csr = _operator(kind, m)
            sv = _factors(csr, case["prec"])
            a = ainv.DeviceOperator(*csr)
            ops.append((csr, sv, a, srv.add_operator(a, sv.device)))
        reqs = []
        for q, xs in enumerate(_solution(case, seed)):
            csr, _, _, op = ops[q % 2]
            b = torch.from_numpy(_csr_times(csr, xs)).pin_memory()
            reqs.append((op, b, torch.empty(len(xs), dtype=torch.float64).pin_memory()))
        return dict(case=case, srv=srv, ops=[o[1:3] for o in ops], reqs=reqs)
    csr = _operator(case["operator"], case["idim"])
    sv = _factors(csr, case["prec"])
    b = torch.from_numpy(np.ascontiguousarray(_csr_times(csr, _solution(case, seed)))).cuda()
    return dict(case=case, a=ainv.DeviceOperator(*csr), sv=sv, f=sv.device, b=b,
                x=torch.zeros_like(b))


def run(state):
    case = state["case"]
    if case["kind"] == "apply":
        state["f"].apply(state["x"], state["y"], case["alpha"], case["beta"], case["trans"])
        return state["y"]
    if case["kind"] == "serve":
        srv = state["srv"]
        ids = [srv.submit(op, b, x, case["eps"], 1000) for op, b, x in state["reqs"]]
        for i in ids:
            srv.wait(i)
        return [x for _, _, x in state["reqs"]]
    state["x"].zero_()
    if case["kind"] == "block":
        state["a"].block_solve(state["b"], state["x"], state["f"], case["eps"], 1000)
        return state["x"]
    r = state["a"].solve(state["b"], state["x"], state["f"], case["method"], case["eps"], 1000)
    return {"x": state["x"], "iter": r.iter}


# ------------------------------------------------------------------ work --
def _nnz(m, stencil):
    total = m ** 3
    for d in stencil:
        total += math.prod(max(0, m - abs(c)) for c in d)
    return total


def work(case):
    """Bytes and operations one pass cannot do without.  An apply reads the
    factors' values, D^-1 and x and writes y (an index per entry where no
    rows share a pattern).  A Krylov iteration reads A and the factors and
    reads and writes its vectors once per step that needs them; the
    iteration counts are those seen on these operators."""
    v = VALUE_BYTES[case["prec"]]

    def precond(m):
        n, nnz = m ** 3, 2 * _nnz(m, AINV_STENCIL)
        return nnz * v + n * v, 2 * nnz + n

    def a_product(m):
        nnz = _nnz(m, [(1, 0, 0), (0, 1, 0), (0, 0, 1)] * 2)
        return nnz * 8, 2 * nnz

    if case["kind"] == "apply":
        n = case["idim"] ** 3
        nnz = 2 * _nnz(case["idim"], INVK_STENCIL if case["pattern"] == "invk" else AINV_STENCIL)
        per = v + (4 if case["pattern"] == "scattered" else 0)
        return {"bytes": nnz * per + n * v + 16 * n + (8 * n if case["beta"] else 0),
                "flops": 2 * nnz + n}

    def krylov(m, method, rhs=1):
        n = m ** 3
        pb, pf = precond(m)
        ab, af = a_product(m)
        if method == "CG":  # x, r, z, p, q: 5 written, 9 read
            its, once, vecs = 2.0 * m, 1, 14
        else:               # x, r, p, v, f, s, z, t: 8 written, 14 read
            its, once, vecs = 1.05 * m, 2, 22
        return (its * (once * (pb + ab) + vecs * 8 * n * rhs),
                its * rhs * (once * (pf + af) + 2 * vecs * n))

    if case["kind"] == "serve":
        b = f = 0.0
        for q in range(case["requests"]):
            got = krylov(case["idim2" if q % 2 else "idim"], "BICGSTAB")
            b, f = b + got[0], f + got[1]
        return {"bytes": b, "flops": f}
    method = "CG" if case["kind"] == "block" else case["method"]
    b, f = krylov(case["idim"], method, case.get("rhs", 1))
    return {"bytes": b, "flops": f}


# ----------------------------------------------------------------- exact --
def exact(case, seed):
    """The product in 64 bits with the factors as given, or the solution
    that the right-hand side was made from."""
    if case["kind"] == "apply":
        wt, z, d, x, y = _apply_inputs(case, seed)
        if case["trans"] == "N":
            r = _csr_times(z, d * _csr_times(wt, x))
        else:
            r = _csr_t_times(wt, d * _csr_t_times(z, x))
        return torch.from_numpy(case["alpha"] * r + (case["beta"] * y if case["beta"] else 0.0))
    s = _solution(case, seed)
    if case["kind"] == "solve":
        return {"x": torch.from_numpy(s), "iter": None}
    return [torch.from_numpy(x) for x in s] if case["kind"] == "serve" else torch.from_numpy(s)


def _csr_t_times(csr, x):
    irp, ja, val = csr
    rows = np.repeat(np.arange(len(irp) - 1), np.diff(irp))
    return np.bincount(ja, weights=val * x[rows], minlength=len(irp) - 1)
