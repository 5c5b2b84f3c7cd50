"""Device memory that a handle holds follows the lists there are: many small systems have short ones."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_small_systems_hold_little(fg):
    rng = np.random.default_rng(1)
    sizes = np.full(4096, 50)
    n = int(sizes.sum())
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.uniform(-1, 1, (n, 1)), device="cuda")
    fg.build_forest(pos[:500].contiguous(), S[:500].contiguous(), sizes[:10], 16, 4, 0.5)  # the library's own data
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    t = fg.build_forest(pos, S, sizes, 16, 4, 0.5)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    per = t.np2p / t.ncells
    assert per < 20 and t.nm2l / t.ncells < 20
    # 2 KB a cell for the walk at first, some 300 bytes a cell and 200 a particle for the rest, scratch as much again
    assert held <= 2 * (2048 + 300) * t.ncells + 2 * 200 * n


def test_growth_gives_the_same_lists(fg):
    """A tree whose lists outgrow the first estimate at several levels, built on a fresh handle, on one with room and
    on one that held a small tree."""
    rng = np.random.default_rng(2)
    n = 60_000
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.uniform(-1, 1, (n, 1)), device="cuda")
    a = fg.build_tree(pos, S, n, 16, 4, 0.4)
    la = [np.sort(x.view("u8,u8"), axis=0) for x in a.lists()]
    assert a.nm2l > 200 * a.ncells and a.np2p > 100 * a.nleaves
    a.rebuild(pos)
    lb = [np.sort(x.view("u8,u8"), axis=0) for x in a.lists()]
    c = fg.build_tree(pos, S, n, n + 1, 4, 0.4)
    assert c.nleaves == 1
    c.ncrit = 16
    c.rebuild(pos)
    lc = [np.sort(x.view("u8,u8"), axis=0) for x in c.lists()]
    for k in range(2):
        assert np.array_equal(la[k], lb[k]) and np.array_equal(la[k], lc[k])
