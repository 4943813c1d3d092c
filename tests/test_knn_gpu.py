"""Nearest-neighbour search of the preconditioner where its list can overflow,
run short of candidates or search many shells: coincident particles, a dense
cluster in a sparse system, lines and a plane (grids of one cell across),
batches of just K + 1 particles, and sizes that leave warps idle.

Squared distances are single precision: three differences of exact inputs
(2^-24 relative each), squared and summed with two more roundings, so a chosen
neighbour may be further than the exact one of its rank by 2 (2 + 2 + 1) 2^-24 <
1e-6 relative.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(rng, K):
    n = 6 * K + 5
    cluster = np.concatenate([rng.normal(0, 0.01, (400, 3)), rng.uniform(-50, 50, (n, 3))])
    same = np.concatenate([np.full((K, 3), 1.5), rng.uniform(0, 3, (300, 3))])
    line = np.zeros((n, 3))
    line[:, K % 3] = rng.uniform(0, 100, n)
    plane = rng.uniform(0, 30, (n, 3))
    plane[:, 2] = 2.0
    return {"cluster": (cluster, 0), "same": (same, 0), "line": (line, 0), "plane": (plane, 0),
            "smallest": (rng.uniform(0, 5, (K + 1, 3)), 0),
            "batches": (rng.uniform(0, 5, (7 * (K + 1), 3)), K + 1)}


@pytest.mark.parametrize("K", [16, 32, 48, 64])
@pytest.mark.parametrize("system", ["cluster", "same", "line", "plane", "smallest", "batches"])
def test_nearest_neighbours(cuda, system, K):
    import torch
    from libmobility_gb300 import _capi
    lib = _capi.load()
    p, nper = _systems(np.random.default_rng(K), K)[system]
    p = p.astype(np.float32)
    N = len(p)
    nper = nper or N
    dp = torch.tensor(p, device="cuda")
    nb = torch.full((K + 1, N), -1, dtype=torch.int32, device="cuda")
    assert lib.lmg_internal_knn_k(K, ctypes.c_void_p(dp.data_ptr()), N, nper,
                                  ctypes.c_void_p(nb.data_ptr()), None) == 0
    torch.cuda.synchronize()
    got = nb.cpu().numpy().T
    q = p.astype(np.float64)
    assert (got[:, 0] == np.arange(N)).all()
    assert (got // nper == (np.arange(N) // nper)[:, None]).all()
    for i in range(N):
        assert len(set(got[i])) == K + 1
        b = i // nper * nper
        ref = np.sort(((q[b:b + nper] - q[i]) ** 2).sum(1))[:K + 1]
        d = ((q[got[i]] - q[i]) ** 2).sum(1)
        assert np.allclose(d, ref, rtol=1e-6, atol=0), i
