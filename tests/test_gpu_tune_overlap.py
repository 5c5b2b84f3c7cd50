"""The overlap switch has two states: 2 is accepted as 1, and the autotuner does not time it twice."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_overlap_states(fg):
    n = 33_000  # every level complete: the tensor-core candidates exist
    rng = np.random.default_rng(1)
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.uniform(-1, 1, (n, 1)), device="cuda")
    t = fg.build_tree(pos, S, n, 128, 6, 0.5)
    table = t.autotune(precision="mixed", reps=1)["table"]
    assert 3 in {c["impl"] for c in table}
    assert {c["overlap"] for c in table} == {0, 1}
    keys = [(c["impl"], c["nslots"], c["grouping"], c["overlap"]) for c in table]
    assert len(keys) == len(set(keys))
    out = []
    for ov in (1, 2):
        t.set_tune(3, 0, 0, ov)
        assert t.get_tune()["overlap"] == ov
        out.append(t.compute_field_fmm(precision="mixed").clone())
    assert torch.equal(out[0], out[1])
