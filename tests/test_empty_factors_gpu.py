"""Factors without entries: the apply is beta * y in every precision, whichever
kernels the layout of an empty matrix leads to."""
import numpy as np
import pytest
import torch

import ainv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["FP64", "FP32", "BF16", "FP32_ACC64", "BF16_ACC64"])
@pytest.mark.parametrize("n", [1, 45, 5000])
def test_apply_scales_y(prec, n):
    none = (np.zeros(n + 1, np.int32), np.zeros(0, np.int32), np.zeros(0))
    f = ainv.DeviceFactors(none, none, np.ones(n), prec=prec)
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    y0 = torch.rand(n, dtype=torch.float64, device="cuda")
    for trans in "NT":
        for beta in (0.0, -0.5):
            y = y0.clone()
            f.apply(x, y, 1.5, beta, trans)
            assert torch.equal(y, beta * y0 + 0.0), (trans, beta)
