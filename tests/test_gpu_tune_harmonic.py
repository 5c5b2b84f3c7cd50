"""The harmonic M2L can be chosen, and is the autotuner's default candidate, for every order and source order it covers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,so", [(1, 0), (12, 0), (2, 1), (9, 1), (12, 1), (3, 2), (12, 2)])
def test_choice_five(fg, p, so):
    n = 4000
    rng = np.random.default_rng(p + so)
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.standard_normal((n, (1, 3, 6)[so])), device="cuda")
    t = fg.build_tree(pos, S, n, 32, p, 0.5, source_order=so)
    ref = t.compute_field_fmm(precision="mixed")
    t.set_tune(5)
    assert t.get_tune()["impl"] == 5
    assert torch.equal(t.compute_field_fmm(precision="mixed"), ref)
    r = t.autotune(precision="mixed", reps=1)
    for c in r["table"]:
        t.set_tune(c["impl"], c["nslots"], c["grouping"], c["overlap"])
    assert {c["impl"] for c in r["table"]} & {0, 5}
    if not (so == 0 and p <= 12 or so == 1 and p <= 8):  # the class-major kernels' range is as it was
        with pytest.raises(fg.FMMError):
            t.set_tune(4)
