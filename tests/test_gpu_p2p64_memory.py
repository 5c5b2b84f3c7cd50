"""The FP64 near field adds in an order that the tree decides: not the memory that is free, and not whether a pass runs
or is captured."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def system(n, so, seed):
    rng = np.random.default_rng(seed)
    return (torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda"),
            torch.tensor(rng.uniform(-1, 1, (n, 1 if so == 0 else 3)), device="cuda"))


def test_free_memory_does_not_matter(fg):
    n = 1_000_000
    pos, S = system(n, 0, 1)
    ref = fg.build_tree(pos, S, n, 128, 3, 0.5).compute_field_fmm(precision="fp64")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    # 14 GB stay free: the shares of this tree (2.6 GB) are more than an eighth of that
    filler = torch.empty(max(free - (14 << 30), 0), dtype=torch.uint8, device="cuda")
    try:
        t = fg.build_tree(pos, S, n, 128, 3, 0.5)
        assert torch.equal(t.compute_field_fmm(precision="fp64"), ref)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert torch.equal(t.compute_field_fmm(precision="fp64"), ref)


@pytest.mark.parametrize("so", [0, 1])
def test_captured_first_pass(fg, so):
    """The first pass of a rebuild captured by the caller, its buffers reserved by the build before."""
    n = 12_000
    pos, S = system(n, so, 2 + so)
    other, _ = system(n, so, 4 + so)
    ref = fg.build_tree(other, S, n, 32, 4, 0.5, source_order=so).compute_field_fmm(precision="fp64")
    t = fg.build_tree(other, S, n, 32, 4, 0.5, source_order=so)
    F = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    t.compute_field_fmm(F, precision="fp64")
    for p in (pos, other):
        t.rebuild(p)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t.compute_field_fmm(F, precision="fp64")
    F.zero_()
    g.replay()
    assert torch.equal(F, ref)
    assert torch.equal(t.compute_field_fmm(precision="fp64"), ref)
