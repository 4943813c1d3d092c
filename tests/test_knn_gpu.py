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


def test_order_of_equal_distances(cuda):
    """On a perfect lattice most distances tie: equal ones come shell by shell of
    the search grid (Chebyshev distance in cells), in the order of the cells'
    coordinates.  The preconditioner's network takes them in this order.  Cells
    are half the expected distance of the 16th neighbour wide, here less than
    the lattice constant, so that no two particles share one."""
    import torch
    from libmobility_gb300 import _capi
    lib = _capi.load()
    K, m = 16, 11
    rng = np.random.default_rng(3)
    p = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.5
    p = p[rng.permutation(m ** 3)].astype(np.float32)
    N = len(p)
    dp = torch.tensor(p, device="cuda")
    nb = torch.empty((K + 1, N), dtype=torch.int32, device="cuda")
    assert lib.lmg_internal_knn_k(K, ctypes.c_void_p(dp.data_ptr()), N, N,
                                  ctypes.c_void_p(nb.data_ptr()), None) == 0
    torch.cuda.synchronize()
    got = nb.cpu().numpy().T
    extent = np.float64(2.5 * (m - 1))
    h = 0.5 * np.cbrt(3 * (K + 1) / (4 * np.pi * N / extent ** 3))
    assert h < 2.5 and np.ceil(extent / h) ** 3 <= 8 * N + 64
    n = int(np.ceil(extent / h))
    cell = np.minimum((p * np.float32(1 / h)).astype(int), n - 1)
    for i in range(N):
        d2 = ((p - p[i]).astype(np.float64) ** 2).sum(1)
        d2[i] = -1
        o = cell - cell[i]
        order = np.lexsort((o[:, 2], o[:, 1], o[:, 0], np.abs(o).max(1), d2))
        assert np.array_equal(got[i], order[:K + 1]), i
