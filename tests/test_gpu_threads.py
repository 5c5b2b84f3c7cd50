"""Trees of different sizes and orders built and evaluated by several threads at once: a kernel's launch limits belong
to the process, so no call may set one that another thread's launch does not fit."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def system(kind, n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0, 1, (n, 3))
    if kind == "deep":
        pos = (pos - 0.5) * rng.uniform(0.02, 1, (n, 1)) ** 1.5
    return torch.tensor(pos, device="cuda"), torch.tensor(rng.uniform(-1, 1, (n, 1)), device="cuda")


def test_builds_side_by_side(fg):
    # many classes (a 64 KB bitmap) and few, long and short rows of the FP64 M2M
    setups = [("deep", 6000, 8, 12), ("uniform", 3000, 32, 11), ("deep", 6000, 8, 11), ("uniform", 3000, 32, 12)]
    args, want = [], []
    for k, (kind, n, ncrit, p) in enumerate(setups):
        pos, S = system(kind, n, k)
        args.append((pos, S, n, ncrit, p))
        want.append(fg.build_tree(pos, S, n, ncrit, p, 0.5).compute_field_fmm(precision="fp64"))
    torch.cuda.synchronize()
    errors = []

    def work(k):
        pos, S, n, ncrit, p = args[k]
        st = torch.cuda.Stream()
        try:
            with torch.cuda.stream(st):
                t = fg.build_tree(pos, S, n, ncrit, p, 0.5)
                for _ in range(60):
                    t.rebuild(pos)
                    F = t.compute_field_fmm(precision="fp64")
                st.synchronize()
                if not torch.equal(F, want[k]):
                    errors.append((k, "fields differ"))
        except Exception as e:  # noqa: BLE001
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(setups))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
