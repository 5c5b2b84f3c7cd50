"""M2L pairs across many levels in the mixed pass: a coarse leaf and a cluster many levels deeper just outside the
distance at which the pair is accepted.  The scaled coefficients of such a pair differ by 2^(degree x levels), beyond
FP32's exponents."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

THETA, NCRIT = 0.5, 8


def system(depth, so, seed=1):
    rng = np.random.default_rng(seed)
    corners = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], float)  # the root cube
    bg = rng.uniform(-0.9, 0.9, (40, 3))
    s = 1.001 / 4  # half-width at level 2
    c = np.array([-3 * s, -s, -s])  # a leaf of level 2, its particles near its corners, the strongest of the system
    own = c + s * np.array([[0.9, 0.9, 0.9], [-0.9, 0.8, -0.9], [0.9, -0.9, -0.8]])
    d = np.array([0.93, 0.2, 0.3])
    shell = c + d / np.linalg.norm(d) * math.sqrt(3) * s / THETA
    cluster = shell + 2.0 ** -depth * rng.uniform(-1, 1, (3000, 3))
    half = np.concatenate([bg, cluster, own])
    pos = np.concatenate([corners, half, -half])
    weight = np.ones(len(pos))
    for first in (8 + 40 + 3000, 8 + 2 * (40 + 3000) + 3):
        weight[first:first + 3] = 1e6
    S = rng.uniform(0.5, 1.5, (len(pos), (1, 3, 6)[so])) * weight[:, None]
    if so == 2:
        S[:, 3] *= -0.5  # not a multiple of the trace, which has no field
    return pos, S


def level(ids):
    return np.array([(int(i).bit_length() - 1) // 3 for i in ids])


def corner_weights(t, p):
    """What a local coefficient adds to the potential at its cell's corner."""
    mi = [(x, y, d - x - y) for d in range(p + 1) for x in range(d, -1, -1) for y in range(d - x, -1, -1)]
    s = t.root()[3] * 0.5 ** level(t.cells()["id"])
    deg = np.array([sum(n) for n in mi])
    fact = np.array([math.factorial(a) * math.factorial(b) * math.factorial(c) for a, b, c in mi], dtype=float)
    return s[:, None] ** deg[None, :] / fact[None, :]


# the last column: levels of difference that the test needs (degree x levels beyond FP32), 0: within FP32 throughout
@pytest.mark.parametrize("so,p,depth,levels", [(0, 12, 10, 11), (0, 12, 14, 14), (0, 9, 14, 15), (0, 8, 14, 16),
                                               (1, 12, 12, 12), (2, 10, 12, 13), (0, 6, 14, 0), (0, 4, 14, 0)])
@pytest.mark.parametrize("orders", [False, True])
def test_locals_across_levels(fg, so, p, depth, levels, orders):
    pos, S = system(depth, so)
    t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), len(pos), NCRIT, p, THETA,
                      source_order=so)
    m2l = t.lists()[0]
    across = level(m2l[:, 1]) - level(m2l[:, 0])
    assert across.max() >= max(levels, 10) and (not levels or p * levels > 126)
    if orders:  # every order up to p among them
        t.set_m2l_orders(np.random.default_rng(3).integers(p - 1, p + 1, t.nm2l).astype(np.uint8))
    w = corner_weights(t, p - so)
    t.compute_field_fmm(precision="fp64")
    L = w * t.expansions()[1]
    choices = [-1] if orders else [-1, 2] + ([4] if so < 1 else [])
    for impl in choices:
        t.set_tune(impl)
        F = t.compute_field_fmm(precision="mixed")
        assert torch.isfinite(F).all()
        Lm = w * t.expansions()[1]
        # each cell's local expansion is a few hundred FP32 terms of FP32 multipoles: 100 roundings of 2^-24
        err, size = np.linalg.norm(Lm - L, axis=1), np.linalg.norm(L, axis=1)
        assert (err <= 100 * 2.0 ** -24 * size).all(), (impl, float((err / np.maximum(size, 1e-300)).max()))
