"""The work that bench.py's roofline figures divide: what the chosen M2L executes, on the CPU."""
import math

import numpy as np
import pytest

import bench
from fmmgen_gb300 import gen_m2l_h as g


@pytest.mark.parametrize("pmax", g.FAMILIES)
def test_multiply_adds_are_the_plan_s(pmax):
    plan = g.plan(pmax)
    for q in range(pmax + 1):
        assert g.multiply_adds(q) == sum(1 for k in plan for t in k["terms"] if t[0] <= q)


def test_m2l_work():
    pairs = 1000
    w = bench.m2l_work(8, pairs, None, 0, 0, None)
    assert "k_m2lh" in w["kernel"] and w["flops"] == 2 * 1365 * pairs
    assert w["cartesian_flops"] == 2 * math.comb(14, 6) * pairs
    for impl in (1, 2, 4):
        w = bench.m2l_work(8, pairs, None, impl, 0, None)
        assert "k_m2lh" not in w["kernel"] and w["flops"] == w["cartesian_flops"]
    assert "tcgen05" in bench.m2l_work(8, pairs, None, 3, 5.0, None)["kernel"]
    orders = np.array([2, 2, 3, 12], np.uint8)
    w = bench.m2l_work(12, 4, orders, -1, 0, {"m2l_multiply_adds": 7})
    assert w["flops"] == 2 * (2 * g.multiply_adds(2) + g.multiply_adds(3) + g.multiply_adds(12))
    assert w["cartesian_flops"] == 14
