"""The root cube's exact sequential FP64 means on sums that keep leaving their binade: the chunk tables, the line
between them and the element scans, and forests, against numpy's sequential accumulation, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def sequential_mean(x):
    return np.add.accumulate(x, axis=0)[-1] / float(len(x))


def column(kind, n, rng):
    if kind == "normal":          # random walk: crossings come in bursts
        return rng.standard_normal(n)
    if kind == "heavy":           # steps of very different sizes
        return rng.standard_normal(n) * 10.0 ** rng.uniform(-6, 2, n)
    if kind == "alternate":       # hovers around a power of two and around zero
        return np.where(np.arange(n) % 2 == 0, 1.0, -1.0) * (1.0 + rng.uniform(0, 1e-3, n))
    if kind == "ties":            # half-ulp terms: the parity of the sum decides
        x = rng.integers(-3, 4, n) * 2.0 ** -53
        x[0] = 1.0
        return x
    if kind == "edges":           # sums that land exactly on powers of two
        return rng.choice([0.25, 0.5, -0.25, -0.5, 1.0, -1.0], n)
    if kind == "tiny":            # subnormal and zero terms
        return rng.choice([0.0, 5e-324, -5e-324, 1e-310], n)
    if kind == "shifted":         # a large offset, then a walk across 2^20
        x = rng.standard_normal(n)
        x[0] = 2.0 ** 20
        return x
    raise ValueError(kind)


KINDS = ["normal", "heavy", "alternate", "ties", "edges", "shifted"]


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 8191, 8192, 8193, 100_003])
@pytest.mark.parametrize("kind", KINDS + ["tiny"])
def test_one_system(fg, kind, n):
    rng = np.random.default_rng(n + KINDS.index(kind) if kind in KINDS else n)
    pos = np.stack([column(kind, n, rng) for _ in range(3)], axis=1)
    if kind == "tiny":
        pos[:, 2] = rng.uniform(0, 1, n)  # a root cube with an extent
    t = fg.build_tree(torch.tensor(pos, device="cuda"), None, n, n + 1, 2, 0.5)
    assert np.array_equal(t.root()[:3], sequential_mean(pos))


@pytest.mark.parametrize("seed", range(4))
def test_two_million(fg, seed):
    rng = np.random.default_rng(seed)
    pos = np.stack([column(k, 2_000_000, rng) for k in ("normal", "heavy", "shifted")], axis=1)
    t = fg.build_tree(torch.tensor(pos, device="cuda"), None, len(pos), len(pos) + 1, 2, 0.5)
    assert np.array_equal(t.root()[:3], sequential_mean(pos))


def test_forest(fg):
    rng = np.random.default_rng(9)
    sizes = [1, 2, 255, 256, 257, 5000, 513, 70_001, 3, 40_000, 1024]
    pos = [np.stack([column(KINDS[(i + a) % len(KINDS)], n, rng) for a in range(3)], axis=1)
           for i, n in enumerate(sizes)]
    f = fg.build_forest(torch.tensor(np.concatenate(pos), device="cuda"), None, sizes, 100_000, 2, 0.5)
    roots, _ = f.systems()
    for p, r in zip(pos, roots):
        assert np.array_equal(r[:3], sequential_mean(p))
