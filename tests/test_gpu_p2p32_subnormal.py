"""FP32 near-field sums below FP32's normal numbers reach the FP64 result: sums of every size, signs, and zeros."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-30, 1e-37, 1e-39, 1e-41, 1e-43])
@pytest.mark.parametrize("n", [2, 7, 40])
def test_small_sums(fg, n, scale):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 1, (n, 3))
    S = rng.uniform(0.5, 1.5, (n, 1)) * scale
    t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), n, 1000, 4, 0.5)
    ref = t.compute_field_fmm(precision="fp64").cpu().numpy()
    F = t.compute_field_fmm(precision="mixed").cpu().numpy()
    d = pos[:, None] - pos[None]
    r = np.sqrt((d ** 2).sum(-1))
    np.fill_diagonal(r, np.inf)
    # a few roundings of each term, of 2^-24 of it or of FP32's smallest number; a term's charge is one of those too
    small = 2.0 ** -149
    tol = 30 * 2.0 ** -24 * (S[:, 0] / r).sum(1) + small * (2 + 1 / r).sum(1)
    assert (np.abs(F[:, 0] - ref[:, 0]) <= tol).all()
    assert (F[:, 0] > 0).all()
    tol = 60 * 2.0 ** -24 * (S[:, 0] / r ** 2).sum(1) + small * (4 + 2 / r + 2 / r ** 2).sum(1)
    assert (np.abs(F[:, 1:] - ref[:, 1:]) <= tol[:, None]).all()
