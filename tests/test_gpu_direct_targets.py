"""Direct sum over a target list with gaps: a negative entry names no particle, is not read and leaves its row of the
output as it is."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("so", [0, 1, 2])
@pytest.mark.parametrize("n,nt", [(40, 3), (700, 33), (5000, 100)])
def test_negative_targets(fg, n, nt, so):
    rng = np.random.default_rng(n + so)
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)), device="cuda")
    S = torch.tensor(rng.uniform(-1, 1, (n, (1, 3, 6)[so])), device="cuda")
    tg = rng.integers(0, n, nt)
    gaps = np.arange(nt) % 3 == 1
    ref = fg.direct(pos, S, targets=tg, source_order=so).cpu().numpy()
    listed = torch.tensor(np.where(gaps, -1 - np.arange(nt), tg), device="cuda")
    F = torch.full((nt, 4), 7.5, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    rc = fg.lib().fmmgen_gpu_direct(C.c_void_p(pos.data_ptr()), C.c_void_p(S.data_ptr()), n,
                                    C.c_void_p(listed.data_ptr()), nt, so, 1, 1, C.c_void_p(F.data_ptr()),
                                    C.c_void_p(st))
    assert rc == 0
    F = F.cpu().numpy()
    assert (F[gaps] == 7.5).all()
    assert np.array_equal(F[~gaps], ref[~gaps])
