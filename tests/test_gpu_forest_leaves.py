"""Forests whose systems are single leaves far below ncrit: the near field's grid follows the particles there are, not
the leaves that ncrit would allow."""
import numpy as np
import pytest
import torch

from test_gpu_p2p64 import close, pairwise

pytestmark = pytest.mark.gpu


# leaves x (largest leaf that ncrit and N allow) / 128 would be 2.2e9 blocks, more than a launch may have
@pytest.mark.parametrize("so", [0, 2])
def test_many_single_leaves(fg, so):
    rng = np.random.default_rng(so)
    nsys = 70_000
    sizes = rng.integers(56, 60, nsys)
    n = int(sizes.sum())
    pos = rng.uniform(0, 1, (n, 3))
    S = rng.uniform(-1, 1, (n, 1 if so == 0 else 6))
    f = fg.build_forest(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), sizes, 5_000_000, so + 1, 0.5,
                        source_order=so)
    assert f.nleaves == nsys and f.nm2l == 0
    F = f.compute_field_fmm(precision="fp64").cpu().numpy()
    off = np.concatenate([[0], np.cumsum(sizes)])
    for s in (0, 1, 2, 3, nsys // 2, nsys - 2, nsys - 1):
        a, b = off[s], off[s + 1]
        ref, mag = pairwise(pos[a:b], S[a:b], so)
        close(F[a:b], ref, mag, b - a)
