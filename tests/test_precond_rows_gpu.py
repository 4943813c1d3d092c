"""P x and P^T x as rows of packed half blocks (the solver's products), where rows of
P^T are long: a row is read 50 entries at a time, so columns with 0, 1, 49, 51, 100
and as many entries as there are particles, and numbers of particles that leave the
last block of eight rows partly empty.  Against the dense products in FP64; an
output of L terms is within (L + 2) u of the sum of its terms' sizes, u = 2^-24.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 48])
@pytest.mark.parametrize("N", [101, 200, 1003])
def test_long_rows(cuda, K, N):
    import torch
    from libmobility_gb300 import _capi
    lib = _capi.load()
    rng = np.random.default_rng(N + K)
    nb = rng.integers(60, N, (K + 1, N)).astype(np.int32)
    nb[0] = np.arange(N)              # the particle itself
    nb[1] = 7                         # a neighbour of all: N entries and its own
    for col, rows in ((11, 48), (12, 50), (13, 99)):
        nb[2 + (col - 11), :rows] = col  # with its own 49, 51 and 100 entries
    blocks = rng.normal(0, 0.3, (K + 1, 9, N)).astype(np.float16)
    x = rng.normal(size=(N, 3)).astype(np.float32)
    B = blocks.astype(np.float64).transpose(0, 2, 1).reshape(K + 1, N, 3, 3)
    xd = x.astype(np.float64)
    want = np.zeros((2, N, 3))
    size = np.zeros((2, N, 3))
    terms = np.zeros((2, N))
    i = np.arange(N)
    for n in range(K + 1):
        t = np.einsum("irc,ic->ir", B[n], xd[nb[n]])
        np.add.at(want[0], i, t)
        np.add.at(size[0], i, np.einsum("irc,ic->ir", abs(B[n]), abs(xd[nb[n]])))
        np.add.at(terms[0], i, 3)
        np.add.at(want[1], nb[n], np.einsum("irc,ir->ic", B[n], xd))
        np.add.at(size[1], nb[n], np.einsum("irc,ir->ic", abs(B[n]), abs(xd)))
        np.add.at(terms[1], nb[n], 3)
    assert {1, 49, 51, 100} <= set((terms[1] / 3).astype(int)) and terms[1].max() >= 3 * N
    d = [torch.tensor(a, device="cuda") for a in (blocks, nb, x)]
    for tr in (0, 1):
        out = torch.full((N, 3), 5.0, device="cuda")  # overwritten
        assert lib.lmg_internal_precond_apply_kh(
            K, ctypes.c_void_p(d[0].data_ptr()), 1, ctypes.c_void_p(d[1].data_ptr()), N,
            ctypes.c_void_p(d[2].data_ptr()), ctypes.c_void_p(out.data_ptr()), tr, None, None) == 0
        torch.cuda.synchronize()
        err = np.abs(out.cpu().numpy() - want[tr])
        assert (err <= (terms[tr][:, None] + 2) * 2.0 ** -24 * size[tr]).all(), tr
