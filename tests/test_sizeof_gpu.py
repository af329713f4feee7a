"""sizeof of device factors against the arrays that they hold."""
import numpy as np
import pytest

import ainv
from util import build_factors, build_inverse_factors, device_factors

pytestmark = pytest.mark.gpu

VALUE = {"FP64": 8, "FP32": 4, "BF16": 2, "FP32_ACC64": 4, "BF16_ACC64": 2}
INTERMEDIATE = {"FP64": 8, "FP32": 4, "BF16": 4, "FP32_ACC64": 8, "BF16_ACC64": 8}


@pytest.mark.parametrize("prec", list(VALUE))
@pytest.mark.parametrize("pattern", ["ainv", "invk", "none"])
def test_covers_every_array(prec, pattern):
    """Per operand: the values, the index words, two row-slice pointers and a
    16-byte word group per slice.  What lies above that is alignment, shared
    offset lists and stage descriptors: no more than the index words of the
    offset slices again, 80 bytes per slice and 256 per array."""
    if pattern == "none":
        n = 700
        none = np.zeros(n + 1, np.int32), np.zeros(0, np.int32), np.zeros(0)
        f = ainv.DeviceFactors(none, none, np.ones(n), prec=prec)
    else:
        csr = ainv.pde.gen_pde3d(20, "convdiff", (3.0, 2.0, -1.0))
        n = 8000
        f = device_factors(build_factors(*csr) if pattern == "ainv"
                           else build_inverse_factors("INVK", *csr), prec)
    vectors = n * (VALUE[prec] + INTERMEDIATE[prec])
    infos = [f.layout_info(w) for w in ("wt", "z", "zt", "w")]
    low = vectors + sum(o["slots"] * VALUE[prec] + o["nidx"] * 4 + o["nslices"] * 24
                        for o in infos)
    high = low + sum(o["nidx"] * 4 + o["nslices"] * 80 + 8 * 256 for o in infos) + 4096
    assert low <= f.sizeof() <= high
