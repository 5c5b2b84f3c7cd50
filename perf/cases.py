"""The measured cases of this framework: what its users have it do, each through a public entry point.

Every case is a dict with a "kind":

  step      build_tree + compute_field_fmm on new positions and sources in one call (`Tree.rebuild_compute`):
            one step of a particle simulation
  eval      `Tree.compute_field_fmm` on a tree that is kept: new sources at fixed positions (FP64 is its default)
  forest    `build_forest` handle, `rebuild_compute`: many independent systems in one call
  learned   `rebuild_compute` with the committed order model attached (per-pair M2L orders)
  demag     `DemagFMM.compute_field_device`: the demagnetising field of a spin lattice
  bh        `Tree.compute_field_bh`: Barnes-Hut on a kept tree
  direct    `direct`: the FP64 pairwise sum
  ops       the batched operators P2M, M2M, M2L, L2L, L2P (and M2P) on caller-owned expansions

The passes that a caller asks for with precision="mixed" compute the far and the near field in FP32 (the tests hold
them to 2e-6 of the FP64 pass), and the simulations that choose them store their fields in FP32: `run` hands those
fields on as float32.  FP64 passes keep float64.
"""
import math

import numpy as np
import torch

import fmmgen_gb300 as fg
from fmmgen_gb300 import learned, operators
from fmmgen_gb300.demag import MU0, DemagFMM

DEV = "cuda"


def listed():
    return [
        # the reference's CPU-sized example as a simulation step: launches and host round trips count
        dict(name="step 1e4 p4", kind="step", n=10_000, p=4, ncrit=64, theta=0.5, so=0, dist="uniform",
             potential=True, precision="mixed"),
        # the benchmark's headline step
        dict(name="step 1e6 p8", kind="step", n=1_000_000, p=8, ncrit=128, theta=0.5, so=0, dist="uniform",
             potential=False, precision="mixed"),
        # dipoles in a Plummer sphere: a deep, adaptive tree
        dict(name="step plummer 2e6 p6", kind="step", n=2_000_000, p=6, ncrit=64, theta=0.5, so=1, dist="plummer",
             potential=True, precision="mixed"),
        # a clustered system of odd size in FP64, where the accuracy of the caller's doubles is wanted
        dict(name="step fp64 clusters 100003 p6", kind="step", n=100_003, p=6, ncrit=64, theta=0.5, so=0,
             dist="mixture", potential=True, precision="fp64"),
        # the reference's own timed region at the headline size: the evaluation alone, in doubles
        dict(name="eval fp64 1e6 p8", kind="eval", n=1_000_000, p=8, ncrit=128, theta=0.5, so=0, dist="uniform",
             potential=True, precision="fp64"),
        # high-order evaluation with FP32 sweeps
        dict(name="eval mixed 3e5 p12", kind="eval", n=300_000, p=12, ncrit=128, theta=0.5, so=0, dist="uniform",
             potential=False, precision="mixed"),
        # many small systems per call (ensembles), sizes log-uniform in [1000, 65536]
        dict(name="forest 512 p6", kind="forest", nsys=512, lo=1000, hi=65536, p=6, ncrit=64, theta=0.5, so=0,
             potential=False),
        # clustered charges at p_max = 12 with the order model
        dict(name="learned 2e6 p12", kind="learned", n=2_000_000, p=12, ncrit=128, theta=0.5),
        # micromagnetics: a film of spins, the tree set up once, one field per time step
        dict(name="demag 120x90x8 p6", kind="demag", nx=120, ny=90, nz=8, p=6, ncrit=64, theta=0.5),
        # the reference's other tree method
        dict(name="bh 1e5 p4", kind="bh", n=100_000, p=4, ncrit=64, theta=0.5, so=0, dist="mixture"),
        # the exact sum a user checks a run against
        dict(name="direct 30011", kind="direct", n=30_011, so=0),
        # the operator surface for programs that own their tree
        dict(name="ops fp64 20000 p8", kind="ops", n=20_000, p=8, so=0, dtype="float64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "eval", "eval", "forest", "learned", "demag", "bh", "direct", "ops",
                       "ops"])
    theta = round(rng.uniform(0.45, 0.6), 3)
    dist = rng.choice(["uniform", "plummer", "mixture"])
    so = rng.choice([0, 0, 1, 2])
    ncrit = rng.choice([32, 48, 64, 100, 128])
    pot = rng.random() < 0.5
    if kind == "step":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        so = min(so, 1) if precision == "mixed" else so
        p = rng.randint(3, 9) if so < 2 else rng.randint(3, 6)
        return dict(kind=kind, n=_log(rng, 3_000, 1_000_000 if precision == "mixed" else 120_000), p=p, ncrit=ncrit,
                    theta=theta, so=so, dist=dist, potential=pot, precision=precision)
    if kind == "eval":
        precision = rng.choice(["mixed", "fp64", "fp64"])
        so = min(so, 1) if precision == "mixed" else so
        p = rng.randint(3, 12 if so == 0 else 8) if so < 2 else rng.randint(3, 6)
        return dict(kind=kind, n=_log(rng, 3_000, 200_000 if precision == "mixed" else 60_000), p=p, ncrit=ncrit,
                    theta=theta, so=so, dist=dist, potential=pot, precision=precision)
    if kind == "forest":
        lo = _log(rng, 300, 3_000)
        return dict(kind=kind, nsys=_log(rng, 8, 256), lo=lo, hi=lo * rng.randint(2, 20), p=rng.randint(3, 8),
                    ncrit=ncrit, theta=theta, so=min(so, 1), potential=pot)
    if kind == "learned":
        return dict(kind=kind, n=_log(rng, 50_000, 1_000_000), p=rng.choice([10, 12]), ncrit=128, theta=0.5)
    if kind == "demag":
        return dict(kind=kind, nx=rng.randint(20, 120), ny=rng.randint(20, 90), nz=rng.randint(1, 10),
                    p=rng.randint(4, 8), ncrit=ncrit, theta=theta)
    if kind == "bh":
        return dict(kind=kind, n=_log(rng, 2_000, 100_000), p=rng.randint(3, 6), ncrit=ncrit, theta=theta,
                    so=min(so, 1), dist=dist)
    if kind == "direct":
        return dict(kind=kind, n=_log(rng, 1_000, 40_000), so=so)
    return dict(kind=kind, n=_log(rng, 100, 40_000), p=rng.randint(3, 10), so=min(so, 1),
                dtype=rng.choice(["float64", "float32"]))


# -- inputs ---------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _positions(g, n, dist):
    if dist == "uniform":
        return _rand(g, n, 3)
    if dist == "plummer":  # scale 0.1, truncated at radius 1
        umax = (1.0 + 0.1 ** 2) ** -1.5
        u = (_rand(g, n) * umax).clamp_min(1e-9)
        r = 0.1 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
        v = _randn(g, n, 3)
        return (v / v.norm(dim=1, keepdim=True) * r[:, None]).contiguous()
    # half uniform in the unit cube, half in 64 Gaussian clusters (sigma 0.01)
    nu = n // 2
    centres = _rand(g, 64, 3)
    which = torch.randint(0, 64, (n - nu,), generator=g, device=DEV)
    return torch.cat([_rand(g, nu, 3), centres[which] + 0.01 * _randn(g, n - nu, 3)])


def _sources(g, n, so):
    return 2.0 * _rand(g, n, 1) - 1.0 if so == 0 else _randn(g, n, 3 if so == 1 else 6)


def _sizes(c):
    """The systems' sizes belong to the case, not to the seed: an ensemble keeps its sizes."""
    r = np.random.default_rng(c["nsys"] * 1_000_003 + c["hi"])
    return np.floor(np.exp(r.uniform(math.log(c["lo"]), math.log(c["hi"]), c["nsys"]))).astype(np.int64)


def _lattice(c):
    i = np.indices((c["nx"], c["ny"], c["nz"])).reshape(3, -1).T
    return np.ascontiguousarray(i, dtype=np.float64) + 0.5


UNIT_LENGTH, MU_S = 1e-9, 1.7e-23  # one-nanometre cells


def _ops_inputs(c, seed):
    g, n, dt = _gen(seed), c["n"], getattr(torch, c["dtype"])
    far = _randn(g, n, 3)
    far = far / far.norm(dim=1, keepdim=True) * (2.0 + 2.0 * _rand(g, n, 1))  # well-separated cells
    near = _rand(g, 3, n, 3) - 0.5
    q = 2.0 * _rand(g, n, 1) - 1.0
    # moments and local coefficients by degree as a unit cell and its well-separated neighbours have them
    deg = torch.tensor([sum(m) for m in _monomials(c["p"])], device=DEV, dtype=torch.float64)
    fact = torch.exp(torch.lgamma(deg + 1.0))
    ms, ls = operators.msize(c["p"], c["so"]), operators.lsize(c["p"], c["so"])
    M = _randn(g, n, ms) * (0.5 ** deg / fact)[len(deg) - ms:]
    L = _randn(g, n, ls) * (fact / 2.5 ** deg)[:ls]
    return {k: v.to(dt).contiguous() for k, v in dict(far=far, d0=near[0], d1=near[1], d2=near[2], q=q, M=M,
                                                      L=L).items()}


def prepare(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    if kind == "ops":
        return dict(case=c, **_ops_inputs(c, seed))
    if kind == "direct":
        return dict(case=c, pos=_rand(g, c["n"], 3), S=_sources(g, c["n"], c["so"]))
    if kind == "demag":
        coords = _lattice(c)
        d = DemagFMM(c["p"], c["ncrit"], c["theta"])
        m = _randn(g, len(coords), 3)
        spin = (m / m.norm(dim=1, keepdim=True)).reshape(-1).contiguous()
        d.setup(coords, np.zeros(3 * len(coords)), MU_S, unit_length=UNIT_LENGTH)
        return dict(case=c, demag=d, spin=spin)
    if kind == "forest":
        sizes = _sizes(c)
        n = int(sizes.sum())
        pos, S = _rand(g, n, 3), _sources(g, n, c["so"])
        tree = fg.build_forest(pos, S, sizes, c["ncrit"], c["p"], c["theta"], source_order=c["so"])
        return dict(case=c, tree=tree, pos=pos, S=S)
    so = c.get("so", 0)
    pos = _positions(g, c["n"], c.get("dist", "mixture"))
    S = _sources(g, c["n"], so)
    tree = fg.build_tree(pos, S, c["n"], c["ncrit"], c["p"], c["theta"], source_order=so)
    s = dict(case=c, tree=tree, pos=pos, S=S)
    if kind == "learned":
        s["model"] = learned.OrderModel.load()
        s["model"].attach(tree)
    return s


# -- one pass -------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "step":
        F = s["tree"].rebuild_compute(s["pos"], S=s["S"], potential=c["potential"], precision=c["precision"])
        return F.float() if c["precision"] == "mixed" else F
    if kind == "eval":
        F = s["tree"].compute_field_fmm(S=s["S"], potential=c["potential"], precision=c["precision"])
        return F.float() if c["precision"] == "mixed" else F
    if kind == "forest":
        return s["tree"].rebuild_compute(s["pos"], S=s["S"], potential=c["potential"], precision="mixed").float()
    if kind == "learned":
        return s["tree"].rebuild_compute(s["pos"], S=s["S"], potential=False, precision="mixed").float()
    if kind == "demag":
        return s["demag"].compute_field_device(s["spin"])
    if kind == "bh":
        return s["tree"].compute_field_bh(S=s["S"])
    if kind == "direct":
        return fg.direct(s["pos"], s["S"], source_order=c["so"])
    return _run_ops(s)


def _run_ops(s):
    c, n, p, so = s["case"], s["case"]["n"], s["case"]["p"], s["case"]["so"]
    out = {}

    def zeros(width):
        return torch.zeros((n, width), dtype=s["far"].dtype, device=DEV)

    ms, ls = operators.msize(p, so), operators.lsize(p, so)
    if so == 0:
        out["P2M"] = zeros(ms)
        operators.P2M_batch(s["d0"], s["q"], out["P2M"], p, so)
    out["M2M"] = zeros(ms)
    operators.M2M_batch(s["d1"], s["M"], out["M2M"], p, so)
    out["M2L"] = zeros(ls)
    operators.M2L_batch(s["far"], s["M"], out["M2L"], p, so)
    out["L2L"] = zeros(ls)
    operators.L2L_batch(s["d1"], s["L"], out["L2L"], p, so)
    out["L2P"] = zeros(4)
    operators.L2P_batch(s["d2"], s["L"], out["L2P"], p, so)
    out["M2P"] = zeros(4)
    operators.M2P_batch(s["far"], s["M"], out["M2P"], p, so)
    return out


# -- what a pass cannot do without ------------------------------------------------
def _fmm_work(n, p, ncrit, so, outsize):
    """A pair of particles costs 20 operations (dipoles 32), a leaf of about ncrit / 3 sees 27 leaves; a cell takes
    about 189 translations, each a contraction of (p + 1)^2 against (p + 1)^2 harmonic coefficients truncated at
    total degree p."""
    leaf = max(1.0, min(float(n), ncrit / 3.0))
    cells = 8.0 / 7.0 * n / leaf
    terms = sum((s + 1) * (2 * s * s + 4 * s + 3) / 3.0 for s in range(p + 1))
    pairs = n * min(float(n), 27.0 * leaf)
    return dict(bytes=8.0 * n * (3 + (1, 3, 6)[so] + outsize),
                flops=(20.0, 32.0, 60.0)[so] * pairs + 2.0 * terms * min(189.0, cells) * cells)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "direct":
        return dict(bytes=8.0 * c["n"] * (3 + (1, 3, 6)[c["so"]] + 4), flops=(20.0, 32.0, 60.0)[c["so"]] * c["n"] ** 2)
    if kind == "ops":
        b = 8 if c["dtype"] == "float64" else 4
        p, so = c["p"], c["so"]
        nt = (p + 1) * (p + 2) * (p + 3) // 6
        shift = math.comb(p + 6, 6)
        return dict(bytes=float(b * c["n"] * (15 + 9 * nt)), flops=float(c["n"] * (3 * 2 * shift + 20 * nt)))
    if kind == "demag":
        return _fmm_work(c["nx"] * c["ny"] * c["nz"], c["p"], c["ncrit"], 1, 3)
    if kind == "forest":
        w = [_fmm_work(int(n), c["p"], c["ncrit"], c["so"], 3 + c["potential"]) for n in _sizes(c)]
        return dict(bytes=sum(x["bytes"] for x in w), flops=sum(x["flops"] for x in w))
    if kind == "bh":
        w = _fmm_work(c["n"], c["p"], c["ncrit"], c["so"], 4)
        nt = (c["p"] + 1) ** 2
        return dict(bytes=w["bytes"], flops=c["n"] * 189.0 * 8.0 * nt)
    return _fmm_work(c["n"], c["p"], c["ncrit"], c.get("so", 0), 3 + c.get("potential", False))


# -- 64-bit values -----------------------------------------------------------------
def _pairwise(pos, S, so):
    """phi, E of every particle from all others, in 64 bits."""
    n = pos.shape[0]
    out = torch.empty((n, 4), dtype=torch.float64, device=pos.device)
    rows = max(1, min(n, 40_000_000 // n))
    if so == 2:
        A = torch.stack([S[:, 0], S[:, 1] / 2, S[:, 2] / 2, S[:, 1] / 2, S[:, 3], S[:, 4] / 2, S[:, 2] / 2, S[:, 4] / 2,
                         S[:, 5]], dim=1).reshape(n, 3, 3)
        tr = (S[:, 0] + S[:, 3] + S[:, 5])[None, :]
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = [pos[a:b, k, None] - pos[None, :, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r2[torch.arange(b - a, device=pos.device), torch.arange(a, b, device=pos.device)] = math.inf
        ri = torch.rsqrt(r2)
        if so == 0:
            w = ri * S[None, :, 0]
            out[a:b, 0] = w.sum(1)
            w = w * ri * ri
            for k in range(3):
                out[a:b, 1 + k] = (w * d[k]).sum(1)
            continue
        r3 = ri * ri * ri
        if so == 1:
            sd = sum(S[None, :, k] * d[k] for k in range(3))
            out[a:b, 0] = -(sd * r3).sum(1)
            w = 3.0 * sd * r3 * ri * ri
            for k in range(3):
                out[a:b, 1 + k] = (S[None, :, k] * r3 - w * d[k]).sum(1)
            continue
        Ad = [sum(A[None, :, i, k] * d[k] for k in range(3)) for i in range(3)]
        rar = sum(Ad[k] * d[k] for k in range(3))
        r5 = r3 * ri * ri
        finite = torch.where(torch.isinf(r2), torch.zeros_like(r2), r2)
        out[a:b, 0] = ((3.0 * rar - tr * finite) * r5).sum(1)
        w = 15.0 * rar * r5 * ri * ri
        for k in range(3):
            out[a:b, 1 + k] = (w * d[k] - 3.0 * r5 * (tr * d[k] + 2.0 * Ad[k])).sum(1)
    return out


def _monomials(p):
    """fmmgen's order of the multi-indices: by degree, then x descending, then y descending."""
    return [(x, y, d - x - y) for d in range(p + 1) for x in range(d, -1, -1) for y in range(d - x, -1, -1)]


def _powers(v, p, mi):
    """v^k / k! of every multi-index."""
    t = [[torch.ones_like(v[:, 0])] for _ in range(3)]
    for a in range(3):
        for k in range(1, p + 1):
            t[a].append(t[a][-1] * v[:, a] / k)
    return torch.stack([t[0][x] * t[1][y] * t[2][z] for x, y, z in mi], dim=1)


def _derivatives(d, p, mi, at):
    """The derivatives of 1/R at d, by the recurrence in the degree."""
    r2 = (d * d).sum(1)
    D = [1.0 / torch.sqrt(r2)]
    for m in mi[1:]:
        k = sum(m)
        v = torch.zeros_like(r2)
        for a in range(3):
            if m[a] >= 1:
                e = list(m)
                e[a] -= 1
                v -= (2 * k - 1) * m[a] * d[:, a] * D[at[tuple(e)]]
            if m[a] >= 2:
                e[a] -= 1
                v -= (k - 1) * m[a] * (m[a] - 1) * D[at[tuple(e)]]
        D.append(v / (k * r2))
    return torch.stack(D, dim=1)


def _ops_exact(c, seed):
    x = {k: v.double() for k, v in _ops_inputs(c, seed).items()}
    p, so, n = c["p"], c["so"], c["n"]
    mi = _monomials(p + 1)
    at = {m: i for i, m in enumerate(mi)}
    nt = {d: sum((k + 1) * (k + 2) // 2 for k in range(d + 1)) for d in range(-1, p + 2)}
    off, top, low = nt[so - 1], nt[p], nt[p - so]

    def add(a, b):
        return at[(a[0] + b[0], a[1] + b[1], a[2] + b[2])]

    def sub(a, b):
        return at.get((a[0] - b[0], a[1] - b[1], a[2] - b[2])) if all(u >= v for u, v in zip(a, b)) else None

    out = {}
    if so == 0:
        out["P2M"] = x["q"] * _powers(-x["d0"], p, mi[:top])
    mono = _powers(x["d1"], p, mi[:top])
    Ms = torch.zeros((n, top - off), dtype=torch.float64, device=DEV)
    for i in range(off, top):
        ks = [(k, sub(mi[i], mi[k])) for k in range(top)]
        ks = [(k, j) for k, j in ks if j is not None and j >= off]
        Ms[:, i - off] = (mono[:, [k for k, _ in ks]] * x["M"][:, [j - off for _, j in ks]]).sum(1)
    out["M2M"] = Ms
    D = _derivatives(x["far"], p + 1, mi, at)
    L = torch.zeros((n, low), dtype=torch.float64, device=DEV)
    for i in range(low):
        js = [j for j in range(off, top) if sum(mi[i]) + sum(mi[j]) <= p]
        L[:, i] = (D[:, [add(mi[i], mi[j]) for j in js]] * x["M"][:, [j - off for j in js]]).sum(1)
    out["M2L"] = L
    Ls = torch.zeros((n, low), dtype=torch.float64, device=DEV)
    for i in range(low):
        ks = [k for k in range(low) if sum(mi[i]) + sum(mi[k]) <= p - so]
        Ls[:, i] = (mono[:, ks] * x["L"][:, [add(mi[i], mi[k]) for k in ks]]).sum(1)
    out["L2L"] = Ls
    mono = _powers(x["d2"], p, mi[:top])
    F = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    F[:, 0] = (x["L"] * mono[:, :low]).sum(1)
    unit = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    for a in range(3):
        ks = [k for k in range(low) if mi[k][a] > 0]
        F[:, 1 + a] = -(x["L"][:, ks] * mono[:, [sub(mi[k], unit[a]) for k in ks]]).sum(1)
    out["L2P"] = F
    F = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    F[:, 0] = (D[:, off:top] * x["M"]).sum(1)
    for a in range(3):
        F[:, 1 + a] = -(D[:, [add(mi[j], unit[a]) for j in range(off, top)]] * x["M"]).sum(1)
    out["M2P"] = F
    return out


def exact(case, seed):
    """The fields are those of the pairwise sum: what the fast methods approximate."""
    c = case
    kind = c["kind"]
    if kind == "ops":
        return _ops_exact(c, seed)
    if kind == "forest":
        sizes = _sizes(c)
        if float((sizes.astype(np.float64) ** 2).sum()) > 3e10:
            return None
        g, n = _gen(seed), int(sizes.sum())
        pos, S = _rand(g, n, 3), _sources(g, n, c["so"])
        off = np.concatenate([[0], np.cumsum(sizes)])
        F = torch.cat([_pairwise(pos[a:b], S[a:b], c["so"]) for a, b in zip(off[:-1].tolist(), off[1:].tolist())])
        return F if c["potential"] else F[:, 1:].contiguous()
    if kind == "demag":
        pos = torch.tensor(_lattice(c), device=DEV)
        g = _gen(seed)
        m = _randn(g, len(pos), 3)
        F = _pairwise(pos, m / m.norm(dim=1, keepdim=True), 1)
        return F[:, 1:] * (-MU0 / (4.0 * math.pi) * MU_S / UNIT_LENGTH ** 3)
    if c["n"] > 310_000:
        return None
    g, so = _gen(seed), c.get("so", 0)
    pos = _rand(g, c["n"], 3) if kind == "direct" else _positions(g, c["n"], c.get("dist", "mixture"))
    F = _pairwise(pos, _sources(g, c["n"], so), so)
    return F if kind in ("bh", "direct") or c.get("potential", False) else F[:, 1:].contiguous()
