"""Registers of the compiled kernels, from the compiler's report of the build."""
import os
import re

import pytest

BUILD = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                     "mld-ainv_b200", "_build")


def spills(name):
    path = os.path.join(BUILD, name + ".ptxas.txt")
    if not os.path.exists(path):
        pytest.skip("no build report here")
    with open(path) as f:
        text = f.read()
    return {k: int(n) for k, n in re.findall(
        r"Function properties for (\S+)\s+\d+ bytes stack frame, (\d+) bytes spill stores", text)}


def test_block_products_keep_their_slots_in_registers():
    got = {k: n for k, n in spills("blockcg").items()
           if re.search("k_mv_(init|spmm_sigma|trueres)", k)}
    assert len(got) == 12 and not any(got.values()), got
