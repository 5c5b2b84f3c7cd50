"""The plan of the harmonic M2L kernels (fmmgen_gb300/gen_m2l_h.py) on the CPU: folding, the kernels' terms and
unfolding together are the full translation, at every truncation order; staged rows and code stay within bounds; the
sources on disk are the generator's."""
import math
import os

import numpy as np
import pytest

from fmmgen_gb300 import gen_m2l_h as g


def monomials(p):
    return [(x, y, d - x - y) for d in range(p + 1) for x in range(d, -1, -1) for y in range(d - x, -1, -1)]


def derivatives(v, p):
    """Derivatives of 1/R by the recurrence in the degree (a harmonic set, as the kernels assume)."""
    D = {}
    r2 = float(v @ v)
    for k in monomials(p):
        d = sum(k)
        if d == 0:
            D[k] = 1 / math.sqrt(r2)
            continue
        s = 0.0
        for a in range(3):
            e = list(k)
            if k[a] >= 1:
                e[a] = k[a] - 1
                s -= (2 * d - 1) * k[a] * v[a] * D[tuple(e)]
            if k[a] >= 2:
                e[a] = k[a] - 2
                s -= (d - 1) * k[a] * (k[a] - 1) * D[tuple(e)]
        D[k] = s / (d * r2)
    return D


@pytest.mark.parametrize("pmax", g.FAMILIES)
@pytest.mark.parametrize("so", [0, 1, 2])
def test_fold_terms_unfold_are_the_translation(pmax, so):
    rng = np.random.default_rng(pmax + so)
    D = derivatives(np.array([2.0, -3.0, 1.5]), pmax)
    mi = monomials(pmax)
    M = {m: (rng.standard_normal() if sum(m) >= so else 0.0) for m in mi}
    co, op = g.coeffs(pmax), g.operators(pmax)
    fold = {}
    for x, y, e in co:
        fold[(x, y, e)] = sum((-1) ** j * math.comb(j, i) * M[(x - 2 * i, y - 2 * (j - i), e + 2 * j)]
                              for j in range((x + y) // 2 + 1) for i in range(j + 1)
                              if 2 * i <= x and 2 * (j - i) <= y)
    for q in range(so + 1, pmax + 1):
        L = np.zeros(len(co))
        for kern in g.plan(pmax):
            if kern["dmin"] > q:
                continue
            for d, k, i, j in kern["terms"]:
                if d <= q:
                    L[i] += D[op[k]] * fold[co[j]]
        at = {n: i for i, n in enumerate(co)}
        for n in monomials(q - so):
            ref = sum(D[(n[0] + m[0], n[1] + m[1], n[2] + m[2])] * M[m] for m in monomials(q - sum(n)))
            e, j = n[2] & 1, n[2] >> 1
            got = (-1) ** j * sum(math.comb(j, i) * L[at[(n[0] + 2 * i, n[1] + 2 * (j - i), e)]] for i in range(j + 1))
            mag = sum(abs(D[(n[0] + m[0], n[1] + m[1], n[2] + m[2])] * M[m]) for m in monomials(q - sum(n)))
            # folding and unfolding add at most a few hundred terms, of binomial weights up to 20
            assert abs(got - ref) <= 1e-11 * (mag + abs(ref)) + 1e-11 * max(abs(v) for v in L), (q, n)


@pytest.mark.parametrize("pmax", g.FAMILIES)
def test_terms_once_and_bounds(pmax):
    seen, stores = set(), set()
    for kern in g.plan(pmax):
        for d, k, i, j in kern["terms"]:
            assert (i, j) not in seen and i in kern["outs"]
            seen.add((i, j))
        if kern["first"]:
            assert not stores & set(kern["outs"])
            stores |= set(kern["outs"])
        else:
            assert set(kern["outs"]) <= stores  # later kernels add to what a first one stored
        assert len(kern["terms"]) <= 1600
        for _, typ, size in g.TYPES:
            mq, dq, split = g.geometry(kern, size)
            assert mq[2] % 2 == 1 and dq[2] % 2 == 1 and dq[0] < split <= dq[1]
            words = mq[2] + dq[2]
            assert 16 * 32 * words * 4 <= g.SMEM                     # four warps of a block fit
            assert len(kern["outs"]) * size <= 16 * words            # the sums fit into the staging area
            per = 16 // size
            assert all(mq[0] <= t[3] // per < mq[1] and dq[0] <= t[1] // per < dq[1] for t in kern["terms"])
    n = g.h_terms(pmax)
    degs = [sum(c) for c in g.coeffs(pmax)]
    assert seen == {(i, j) for i in range(n) for j in range(n) if degs[i] + degs[j] <= pmax}
    assert stores == set(range(n))


def test_generated_sources_are_current(tmp_path, monkeypatch):
    disk = {os.path.basename(f): open(f).read() for f in g.outputs()}
    monkeypatch.setattr(g, "CSRC", str(tmp_path))
    g.generate()
    for name, text in disk.items():
        assert open(os.path.join(tmp_path, name)).read() == text, name
