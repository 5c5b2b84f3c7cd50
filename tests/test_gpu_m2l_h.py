"""M2L over harmonic coefficients (csrc/m2l_h*.cu), FP64 and FP32, against the contraction engine's full translation:
every family and its edges, every source order, per-pair orders, trees of few and of many cells (the lists split over
warps and clusters), lists of unequal length and pairs across levels."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def system(kind, n, so, seed):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        pos = rng.uniform(0, 1, (n, 3))
    else:
        r = 0.1 / np.sqrt(rng.uniform(0.01, 1.0, n) ** (-2.0 / 3.0) - 1.0)
        v = rng.standard_normal((n, 3))
        pos = v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]
    S = rng.uniform(-1, 1, (n, 1)) if so == 0 else rng.standard_normal((n, 3 if so == 1 else 6))
    return torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda")


def locals_of(t, precision):
    t.compute_field_fmm(precision=precision)
    return t.expansions()[1]


def corner_weights(t, p):
    """What a local coefficient adds to the potential at its cell's corner: s^|n| / n! (cells in export order)."""
    mi = [(x, y, d - x - y) for d in range(p + 1) for x in range(d, -1, -1) for y in range(d - x, -1, -1)]
    level = np.array([(int(i).bit_length() - 1) // 3 for i in t.cells()["id"]])
    s = t.root()[3] * 0.5 ** level
    deg = np.array([sum(n) for n in mi])
    fact = np.array([math.factorial(a) * math.factorial(b) * math.factorial(c) for a, b, c in mi], dtype=float)
    return s[:, None] ** deg[None, :] / fact[None, :]


@pytest.mark.parametrize("so,p", [(0, 1), (0, 4), (0, 5), (0, 6), (0, 7), (0, 8), (0, 9), (0, 12), (1, 2), (1, 6),
                                  (1, 9), (1, 12), (2, 3), (2, 6), (2, 10)])
@pytest.mark.parametrize("kind,n,ncrit", [("uniform", 700, 20), ("plummer", 6000, 32)])
def test_locals_match_the_engine(fg, kind, n, ncrit, so, p):
    pos, S = system(kind, n, so, 17 * p + so)
    t = fg.build_tree(pos, S, n, ncrit, p, 0.5, source_order=so)
    assert t.nm2l > 0
    L = locals_of(t, "fp64")
    Lm = locals_of(t, "mixed")
    t.set_tune(impl=2)
    ref = locals_of(t, "fp64")
    Lme = locals_of(t, "mixed")
    # the same sums in another order, FP64: as the operators' tolerance
    assert rel(L, ref) < 1e-12
    # FP32: no worse than twice the engine's own distance, or FP32 rounding of a few hundred terms, in what the
    # coefficients add to the potential (unfolding rounds the highest degrees against each other, whose share of it
    # is the smallest)
    w = corner_weights(t, p - so)
    assert rel(w * Lm, w * ref) < max(2 * rel(w * Lme, w * ref), 1e-6)
    # every cell, not only the large ones: each row against its own size
    a, b = np.linalg.norm(L - ref, axis=1), np.linalg.norm(ref, axis=1)
    assert (a <= 1e-11 * b + 1e-12 * b.max() * 1e-6).all()


def test_many_cells(fg):
    """More targets than the split rule's limit: one block per 32 targets."""
    pos, S = system("uniform", 400_000, 0, 3)
    t = fg.build_tree(pos, S, 400_000, 24, 3, 0.5)
    assert t.ncells > 28 * 152 * 32 / 8
    L = locals_of(t, "fp64")
    t.set_tune(impl=2)
    assert rel(L, locals_of(t, "fp64")) < 1e-12


@pytest.mark.parametrize("so,p", [(0, 8), (0, 12), (1, 5), (2, 6)])
def test_pair_orders_fp64(fg, so, p):
    pos, S = system("plummer", 5000, so, 90 + p)
    t = fg.build_tree(pos, S, 5000, 32, p, 0.5, source_order=so)
    t.set_m2l_orders(np.random.default_rng(p).integers(0, p + 2, t.nm2l).astype(np.uint8))
    L = locals_of(t, "fp64")
    t.set_tune(impl=2)
    assert rel(L, locals_of(t, "fp64")) < 1e-12


def test_rebuild_and_grouping(fg):
    """The target order follows a rebuild and the cell grouping; per-pair orders in between do not leave theirs."""
    pos, S = system("plummer", 5000, 0, 5)
    other, _ = system("uniform", 5000, 0, 6)
    t = fg.build_tree(pos, S, 5000, 32, 6, 0.5)
    ref = t.compute_field_fmm(precision="fp64").cpu().numpy()
    t.set_m2l_orders(np.full(t.nm2l, 3, np.uint8))
    t.compute_field_fmm(precision="fp64")
    t.set_m2l_orders(None)
    assert np.array_equal(t.compute_field_fmm(precision="fp64").cpu().numpy(), ref)
    t.set_tune(-1, 0, 1, 0)
    assert rel(t.compute_field_fmm(precision="fp64").cpu().numpy(), ref) < 1e-12
    t.set_tune(-1, 0, 0, 0)
    t.rebuild(other)
    fresh = fg.build_tree(other, S, 5000, 32, 6, 0.5)
    assert np.array_equal(t.compute_field_fmm(precision="fp64").cpu().numpy(),
                          fresh.compute_field_fmm(precision="fp64").cpu().numpy())
