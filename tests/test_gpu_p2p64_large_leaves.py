"""FP64 near field of trees of few large leaves: a leaf's targets are shared out among warps, whatever the choice between
each pair once and one way, on both sides of the rule's line."""
import numpy as np
import pytest
import torch

from test_gpu_p2p64 import close, pairwise, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("so", [0, 1])
@pytest.mark.parametrize("n,ncrit", [(3000, 5000), (3000, 1000), (3000, 100), (2500, 40), (700, 300)])
def test_sums(fg, n, ncrit, so):
    pos, S = system(n, so, n + so + ncrit)
    t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), n, ncrit, 4, 1e-3,
                      source_order=so)
    assert t.nm2l == 0
    F = t.compute_field_fmm(precision="fp64")
    ref, mag = pairwise(pos, S, so)
    close(F.cpu().numpy(), ref, mag, n)
    assert torch.equal(t.compute_field_fmm(precision="fp64"), F)
    E = t.compute_field_fmm(precision="fp64", potential=False).cpu().numpy()
    close(E, ref[:, 1:], mag[:, 1:], n)
    assert torch.equal(t.rebuild_compute(precision="fp64"), F)


def test_one_large_leaf_fills_the_gpu(fg):
    """16,000 particles in one leaf: 2.6e8 interactions, 18 ms when shared out and more than five seconds by one warp."""
    n = 16_000
    pos, S = system(n, 0, 1)
    t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), n, 2 * n, 4, 0.5)
    assert t.nleaves == 1
    t.compute_field_fmm(precision="fp64")
    assert t.kernel_ms()["P2P"] < 500
