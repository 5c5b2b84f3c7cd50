"""FP32 near field where its work splits change: leaves of every remainder of a chunk of 32 targets (lanes per target
2, 4, 8), source streams around the staged chunk of 64, and source leaves around the far rule's line (a target-leaf
width away), against the FP64 pass."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def system(n, so, seed, box=1.0):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, box, (n, 3)), rng.uniform(-1, 1, (n, 1 if so == 0 else 3))


def fields(fg, pos, S, so, ncrit, p=4, scale=1.0):
    t = fg.build_tree(torch.tensor(pos * scale, device="cuda"), torch.tensor(S, device="cuda"), len(pos), ncrit, p,
                      0.5, source_order=so)
    a = t.compute_field_fmm(precision="fp64").cpu().numpy()
    b = t.compute_field_fmm(precision="mixed").cpu().numpy()
    e = t.compute_field_fmm(precision="mixed", potential=False).cpu().numpy()
    return t, a, b, e


def magnitudes(pos, S, so):
    """Sums of the magnitudes of a particle's interactions (potential, field): what rounding is relative to."""
    d = pos[:, None] - pos[None]
    r = np.sqrt((d ** 2).sum(-1))
    np.fill_diagonal(r, np.inf)
    s = np.abs(S[None, :, 0]) if so == 0 else np.linalg.norm(S, axis=1)[None]
    return (s / r ** (1 + so)).sum(1), (s / r ** (2 + so)).sum(1)


@pytest.mark.parametrize("so", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 24, 25, 31, 32, 33, 40, 48, 63, 64, 65, 66, 127, 129, 500])
def test_one_leaf(fg, n, so):
    pos, S = system(n, so, 7 * n + so)
    t, a, b, e = fields(fg, pos, S, so, 1000)
    assert t.nleaves == 1
    if n == 1:
        assert (b == 0).all() and (e == 0).all()
        return
    mp, mf = magnitudes(pos, S, so)
    # an interaction: about 12 FP32 roundings and a reciprocal square root of 2^-22.9; dipoles' terms reach 4 s / r^3
    tol = (1 + 3 * so) * (12 * 2.0 ** -24 + 3 * 2.0 ** -22)
    assert (np.abs(a[:, 0] - b[:, 0]) <= tol * mp).all()
    assert (np.linalg.norm(a[:, 1:] - b[:, 1:], axis=1) <= 2 * tol * mf).all()
    assert (np.linalg.norm(a[:, 1:] - e, axis=1) <= 2 * tol * mf).all()


# dipoles in a box of 1e-9 leave FP32's range in the mixed pass (1/r^5 of close pairs): charges only
@pytest.mark.parametrize("so,scale", [(0, 1.0), (0, 1e-9), (0, 1e6), (1, 1.0), (1, 1e6)])
def test_far_rule(fg, so, scale):
    """Two clumps of particles in leaves next to each other, a leaf apart and further, on either side of the line; and
    leaves of different levels.  The far frame must not cost accuracy."""
    rng = np.random.default_rng(11 + so)
    clumps = [np.array([x, y, z]) for x in (0.06, 0.19, 0.31, 0.44, 0.94) for y in (0.06, 0.31) for z in (0.06, 0.56)]
    pos = np.concatenate([c + 0.05 * rng.uniform(-1, 1, (int(k), 3)) for c, k in zip(clumps, rng.integers(3, 60, 20))]
                         + [rng.uniform(0, 1, (40, 3))])
    S = rng.uniform(-1, 1, (len(pos), 1 if so == 0 else 3))
    t, a, b, e = fields(fg, pos, S, so, 24, p=10, scale=scale)
    assert t.nleaves > 20
    mp, mf = magnitudes(pos * scale, S, so)
    tol = (1 + 3 * so) * (12 * 2.0 ** -24 + 3 * 2.0 ** -22)
    assert (np.abs(a[:, 0] - b[:, 0]) <= tol * mp).all()
    assert (np.linalg.norm(a[:, 1:] - b[:, 1:], axis=1) <= 2 * tol * mf).all()
    assert np.array_equal(b[:, 1:], e)
