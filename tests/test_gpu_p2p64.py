"""FP64 near field and direct sum at the sizes where their work splits change: leaves of every remainder class of
the target groups (32, 16, 8, the last m <= 7), source streams around the staged chunk, and target counts around a
warp.  A system smaller than ncrit is one leaf, so its FMM is the near field alone."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SS = {0: 1, 1: 3, 2: 6}


def pairwise(pos, S, so, targets=None):
    """phi, E in float64 (long double sums)."""
    t = np.arange(len(pos)) if targets is None else np.asarray(targets)
    d = pos[t, None, :] - pos[None, :, :]
    r2 = (d ** 2).sum(-1)
    r2[np.arange(len(t)), t] = np.inf
    r = np.sqrt(r2)
    if so == 0:
        phi = S[None, :, 0] / r
        E = (S[None, :, 0] / r ** 3)[..., None] * d
    elif so == 1:
        sd = (S[None] * d).sum(-1)
        phi = -sd / r ** 3
        E = S[None] / (r ** 3)[..., None] - (3 * sd / r ** 5)[..., None] * d
    else:
        A = np.array([[S[:, 0], S[:, 1] / 2, S[:, 2] / 2], [S[:, 1] / 2, S[:, 3], S[:, 4] / 2],
                      [S[:, 2] / 2, S[:, 4] / 2, S[:, 5]]]).transpose(2, 0, 1)
        Ad = np.einsum("jab,ijb->ija", A, d)
        rar = (Ad * d).sum(-1)
        tr = np.trace(A, axis1=1, axis2=2)[None]
        r2f = np.where(np.isinf(r2), 0.0, r2)
        phi = (3 * rar - tr * r2f) / r ** 5
        E = (15 * rar / r ** 7)[..., None] * d - 3 / (r ** 5)[..., None] * (tr[..., None] * d + 2 * Ad)
    out = np.concatenate([phi[..., None], E], axis=-1).astype(np.longdouble).sum(1)
    # the sum of magnitudes scales the rounding of any summation order
    mag = np.abs(np.concatenate([phi[..., None], E], axis=-1)).sum(1)
    return out.astype(np.float64), mag


def system(n, so, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, 1, (n, 3)), rng.uniform(-1, 1, (n, SS[so]))


def close(F, ref, mag, n):
    # a term is a chain of ~30 roundings, the sum adds at most n; twice that
    assert (np.abs(F - ref) <= 2 * (30 + n) * 2.2e-16 * mag + 1e-300).all()


@pytest.mark.parametrize("so", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 7, 8, 9, 15, 16, 17, 23, 24, 31, 32, 33, 56, 63, 64, 65, 97, 300])
def test_one_leaf(fg, n, so):
    pos, S = system(n, so, 10 * n + so)
    t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), n, 1000, 4, 0.5,
                      source_order=so)
    assert t.nleaves == 1
    ref, mag = pairwise(pos, S, so)
    F = t.compute_field_fmm(precision="fp64").cpu().numpy()
    close(F, ref, mag, n)
    E = t.compute_field_fmm(precision="fp64", potential=False).cpu().numpy()
    close(E, ref[:, 1:], mag[:, 1:], n)


@pytest.mark.parametrize("so", [0, 1, 2])
@pytest.mark.parametrize("n,nt", [(1, 1), (63, 2), (64, 5), (65, 31), (513, 32), (2000, 33), (2000, None), (9000, 3),
                                  (9000, 700), (4095, None), (4096, None), (4097, None), (4640, None), (5200, None)])
def test_direct(fg, n, nt, so):
    pos, S = system(n, so, n + so)
    tg = None if nt is None else np.random.default_rng(3).integers(0, n, nt)
    ref, mag = pairwise(pos, S, so, tg)
    tt = None if tg is None else torch.tensor(tg)
    P, Q = torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda")
    close(fg.direct(P, Q, targets=tt, source_order=so).cpu().numpy(), ref, mag, n)
    close(fg.direct(P, Q, targets=tt, source_order=so, field=False).cpu().numpy(), ref[:, :1], mag[:, :1], n)
    close(fg.direct(P, Q, targets=tt, source_order=so, potential=False).cpu().numpy(), ref[:, 1:], mag[:, 1:], n)


@pytest.mark.parametrize("so", [0, 1])
@pytest.mark.parametrize("n,ncrit,kind", [(300, 10, "uniform"), (900, 40, "plummer"), (1500, 70, "uniform"),
                                          (2500, 130, "plummer"), (1200, 3, "uniform")])
def test_pairs_once(fg, n, ncrit, kind, so):
    """Trees of leaves of every group size, each pair of leaves worked off once by its owner: with theta so small that
    no pair of cells is well separated the FMM is the pairwise sum; the same bits in every pass, and for the field
    alone."""
    pos, S = system(n, so, n + so)
    if kind == "plummer":
        pos = (pos - 0.5) * np.random.default_rng(n).uniform(0.01, 1, (n, 1)) ** 3
    t = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), n, ncrit, 4, 1e-3,
                      source_order=so)
    assert t.nleaves > 8 and t.nm2l == 0
    ref, mag = pairwise(pos, S, so)
    F = t.compute_field_fmm(precision="fp64")
    close(F.cpu().numpy(), ref, mag, n)
    assert torch.equal(t.compute_field_fmm(precision="fp64"), F)
    assert torch.equal(t.compute_field_fmm(precision="fp64", potential=False), F[:, 1:])
    fresh = fg.build_tree(torch.tensor(pos, device="cuda"), torch.tensor(S, device="cuda"), n, ncrit, 4, 1e-3,
                          source_order=so)
    assert torch.equal(fresh.rebuild_compute(precision="fp64"), F)
