"""Calls of one handle on several streams, none of which the caller orders: a call
uses the handle's buffers after the calls before it, so the results are those of
one stream, bit for bit.  Small systems, whose kernels would fit on the GPU
together; positions set on one stream and used on another; host arrays (the
handle's own stream) beside device arrays.
"""
import numpy as np
import pytest

from test_mdot_gpu import make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("wall,ang", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("N", [40, 200, 700])
def test_calls_follow_each_other(cuda, precision, wall, ang, N):
    import torch
    rng = np.random.default_rng(N + 2 * wall + ang)
    dt = torch.float32 if precision == "float" else torch.float64
    side = (N * 4 * np.pi / 3 / 0.15) ** (1 / 3)
    P = [torch.tensor(rng.uniform(0, side, (N, 3)) + 0.5, dtype=dt, device="cuda")
         for _ in range(4)]
    F = torch.tensor(rng.normal(size=(32, N, 3)), dtype=dt, device="cuda")
    T = torch.tensor(rng.normal(size=(32, N, 3)), dtype=dt, device="cuda")

    def calls(s, streams):
        out = []
        for k in range(32):
            with torch.cuda.stream(streams[k % len(streams)]):
                if k % 8 == 0:
                    s.setPositions(P[k // 8])
                if k % 8 == 5:  # host arrays: the handle's own stream
                    out += [torch.tensor(x) for x in s.Mdot(F[k].cpu().numpy()) if x is not None]
                elif k % 8 == 6 and wall:
                    s.divM(1.0)  # leaves work and draws noise, the same either way
                else:
                    out += [x for x in s.Mdot(F[k], T[k] if ang else None) if x is not None]
        torch.cuda.synchronize()
        return [x.cpu() for x in out]

    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    want = calls(make_solver(wall, ang, 1.0, 1.0, precision), streams[:1])
    got = calls(make_solver(wall, ang, 1.0, 1.0, precision), streams)
    assert len(got) == len(want)
    for k, (x, y) in enumerate(zip(got, want)):
        assert torch.equal(x, y), k


def test_a_stream_may_be_gone(cuda):
    """The stream of the last call need not exist any more."""
    import ctypes

    import torch
    from libmobility_gb300 import _capi
    rt = ctypes.CDLL("libcudart.so.13", mode=ctypes.RTLD_GLOBAL)
    s = make_solver(1, 1, 1.0, 1.0, "float")
    rng = np.random.default_rng(0)
    p, F, T = (torch.tensor(x, dtype=torch.float32, device="cuda")
               for x in (rng.uniform(1, 9, (100, 3)), *rng.normal(size=(2, 100, 3))))
    U, W = torch.empty((2, 100, 3), device="cuda")
    s.setPositions(p)
    want = s.Mdot(F, T)
    torch.cuda.synchronize()
    lib, h = _capi.load(), s._h
    for _ in range(3):
        st = ctypes.c_void_p()
        assert rt.cudaStreamCreate(ctypes.byref(st)) == 0
        assert lib.lmg_set_stream(h, st) == 0
        assert lib.lmg_mdot(h, F.data_ptr(), 300, T.data_ptr(), 300, U.data_ptr(), 300,
                            W.data_ptr(), 300) == 0
        assert rt.cudaStreamDestroy(st) == 0
    got = s.Mdot(F, T)
    torch.cuda.synchronize()
    for x, y in zip((*got, U, W), (*want, *want)):
        assert torch.equal(x, y)
