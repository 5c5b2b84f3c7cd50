"""A recorded evaluation pass keeps its buffers: calls on the same tree in between that work in another precision, or
by Barnes-Hut, must not move them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def tree(fg, n, p, so=0):
    rng = np.random.default_rng(100 * p + so)
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.uniform(-1, 1, (n, (1, 3, 6)[so])), device="cuda")
    return fg.build_tree(pos, S, n, 32, p, 0.5, source_order=so)


# orders at which a Barnes-Hut row of 8 (p + 1)^2 bytes is longer than the padded FP32 row of the M2L, and one where not
@pytest.mark.parametrize("p,so", [(4, 0), (5, 0), (6, 1), (8, 0), (12, 0), (4, 2)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_barnes_hut_between_replays(fg, p, so, precision):
    n = 8000
    t = tree(fg, n, p, so).set_graph(True)
    F = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    t.compute_field_fmm(F, precision=precision)  # recorded
    ref = F.clone()
    bh = t.compute_field_bh().clone()
    other = torch.zeros(1 << 22, device="cuda")  # memory that a freed buffer's pages could have gone to
    F.zero_()
    t.compute_field_fmm(F, precision=precision)  # replayed
    assert torch.equal(F, ref)
    assert not other.any()
    assert torch.equal(t.compute_field_bh(), bh)


@pytest.mark.parametrize("p,so", [(4, 0), (8, 0), (7, 1)])
def test_other_precision_between_replays(fg, p, so):
    """The pass captured by the caller: nothing tells the tree that it is replayed later."""
    n = 8000
    t = tree(fg, n, p, so)
    F = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    t.compute_field_fmm(F, precision="mixed")
    ref = F.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t.compute_field_fmm(F, precision="mixed")
    t.compute_field_fmm(precision="fp64")
    t.compute_field_bh()
    F.zero_()
    g.replay()
    assert torch.equal(F, ref)
