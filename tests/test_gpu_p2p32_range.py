"""The FP32 near field holds positions as two FP32 numbers an axis, between leaves that do not touch as well: every
component of a displacement keeps its own relative accuracy.  A coordinate rounded to one FP32 number, in a frame as wide
as the distance, would lose the small components."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("so", [0, 1])
@pytest.mark.parametrize("ncrit", [2, 3, 10, 40])
@pytest.mark.parametrize("gap", [2.0 ** -2, 2.0 ** -4, 2.0 ** -8])
def test_small_components(fg, gap, ncrit, so):
    n = 16
    rng = np.random.default_rng(int(1 / gap) + so)
    base = rng.uniform(0, 0.25, (n, 3))
    d = gap * np.stack([rng.uniform(1, 2, n), 2.0 ** -7 * rng.uniform(-1, 1, n), 2.0 ** -14 * rng.uniform(0.5, 1, n)], 1)
    pos = np.concatenate([base, base + d])
    for k in range(n):  # one source at a time, its partner's field
        S = np.zeros((2 * n, 1 if so == 0 else 3))
        S[k] = 1.0 if so == 0 else (1.0, 0.0, 0.0)  # along x: the small components are -3 x (y, z) / r^5
        t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), 2 * n, ncrit, 4, 1e-3,
                          source_order=so)
        assert t.nm2l == 0  # nothing is far enough for so small a theta: the near field alone
        F = t.compute_field_fmm(precision="mixed").cpu().numpy()[n + k]
        x = pos[n + k] - pos[k]
        r = np.linalg.norm(x)
        E = x / r ** 3 if so == 0 else S[k] / r ** 3 - 3 * x[0] * x / r ** 5
        # a displacement: two roundings; r^2: three more; its reciprocal root 2^-22.9 and up to its fifth power; products
        tol = ((2 + 5 * (2 + 1.5) + 5 * 2.2 + 5) * (1 if so == 0 else 2)) * 2.0 ** -24
        assert (np.abs(F[1:] - E) <= tol * np.abs(E)).all(), (k, (F[1:] - E) / E * 2.0 ** 24)
