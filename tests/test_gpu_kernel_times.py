"""The kernels' own times are the last pass's, also where a pass has no M2L pairs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_pairs_no_time(fg, precision):
    rng = np.random.default_rng(1)
    n = 20_000
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.uniform(-1, 1, (n, 1)), device="cuda")
    t = fg.build_tree(pos, S, n, 16, 12, 0.4)
    t.compute_field_fmm(precision=precision)
    before = t.kernel_ms()["M2L"]
    assert t.nm2l > 1_000_000 and before > 0.2
    t.ncrit = n + 1
    t.rebuild(pos)
    t.compute_field_fmm(precision=precision)
    assert t.nm2l == 0 and t.kernel_ms()["M2L"] < 0.5 * before
