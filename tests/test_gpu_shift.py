"""M2M and L2L along the axes (csrc/shift.cu): every cell's expansions against the restatement of the reference, with
children missing, far from the origin, at the orders' ends."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.tensor(a, device="cuda")


def degrees(lo, hi):
    return np.concatenate([np.full((d + 1) * (d + 2) // 2, d) for d in range(lo, hi + 1)])


@pytest.mark.parametrize("so,p,kind", [(0, 1, "uniform"), (0, 4, "cluster"), (0, 8, "shell"), (0, 12, "uniform"),
                                       (1, 2, "shell"), (1, 7, "cluster"), (2, 3, "uniform"), (2, 8, "shell"),
                                       (0, 5, "far")])
def test_expansions(fg, oracle_lib, so, p, kind):
    rng = np.random.default_rng(10 * p + so)
    n = 1500
    pos = rng.uniform(-1, 1, (n, 3))
    if kind == "cluster":
        pos *= rng.uniform(0.02, 1, (n, 1)) ** 2
    if kind == "shell":
        pos /= np.linalg.norm(pos, axis=1, keepdims=True)
    if kind == "far":
        pos += 1e5
    S = rng.uniform(-1, 1, (n, [1, 3, 6][so]))
    t = fg.build_tree(cuda(pos), cuda(S), n, 24, p, 0.5, source_order=so)
    assert t.nlevels > 3
    t.compute_field_fmm(precision="fp64")
    M, L = t.expansions()
    t.compute_field_fmm(precision="mixed")
    Mf, _ = t.expansions()
    ot = oracle_lib.OracleTree(pos, S, 24, p, 0.5, so)
    _, _, Mo, Lo = ot.evaluate(want_ML=True)
    row = {int(i): k for k, i in enumerate(ot.cells()["id"])}
    c = t.cells()
    perm = np.array([row[int(i)] for i in c["id"]])
    # far from the origin the particles' offsets from a centre carry 1e5 ulps of the cell's size
    tol = 1e-10 if kind != "far" else 1e-8
    for a, b in ((M, Mo[perm]), (L, Lo[perm])):
        assert np.max(np.abs(a - b).max(axis=1) / np.maximum(np.abs(b).max(axis=1), 1e-300)) < tol
    # FP32: a few levels of three sums of up to p + 1 terms, each rounded to 6e-8, in units of the cell
    s = np.abs(pos - pos.mean(0)).max() * 1.001 * 0.5 ** ((np.array([int(i).bit_length() for i in c["id"]]) - 1) // 3)
    scale = s[:, None] ** -degrees(so, p)[None].astype(float)
    a, b = Mf * scale, M * scale
    assert np.max(np.abs(a - b).max(axis=1) / np.abs(b).max(axis=1)) < 1e-5
