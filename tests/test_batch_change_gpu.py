"""One handle whose batches change while N stays (setParameters and setPositions
without initialize): products and square roots are those of a handle made for
the new batches, bit for bit, and agree with the FP64 oracle (1e-5 and 1e-12
relative, as every Mdot).  A launch plan's splits cover the sources of a tile's
batches, so one made for small batches is too short for large ones.
"""
import numpy as np
import pytest

from test_mdot_gpu import make_solver, rel_err

pytestmark = pytest.mark.gpu
TOL = {"float": 1e-5, "double": 1e-12}


@pytest.fixture()
def lib(cuda):
    from libmobility_gb300 import _capi
    lib = _capi.load()
    yield lib
    lib.lmg_internal_sym_override(0, 0)


@pytest.mark.parametrize("order", [(100, 1000, 100), (1000, 100, 1000), (250, 500, 1000)])
@pytest.mark.parametrize("precision,wall,ang", [("float", 1, 0), ("float", 1, 1), ("float", 0, 1),
                                                ("double", 0, 0), ("double", 1, 1)])
@pytest.mark.parametrize("mode", [0, 1])  # 1: Mdot takes mdot_kernel too
def test_batches_change_at_the_same_n(lib, oracle, order, precision, wall, ang, mode):
    rng = np.random.default_rng(5)
    N = 1000
    p = rng.uniform(0, (N * 4 * np.pi / 3 / 0.05) ** (1 / 3), (N, 3))
    if wall:
        p[:, 2] = rng.uniform(1.5, 10, N)
    F, T = rng.normal(size=(2, N, 3))
    T = T if ang else None
    dW = rng.normal(size=N * (6 if ang else 3))
    p, F, dW = (x.astype(np.float32 if precision == "float" else np.float64) for x in (p, F, dW))
    T = None if T is None else T.astype(F.dtype)
    assert lib.lmg_internal_sym_override(mode, 0) == 0

    def handle(nper):
        h = make_solver(wall, ang, 1.0, 1.0, precision, N, nper)
        # with a callback every iteration is checked: solves before this one have no say
        h.initialize(viscosity=1.0, hydrodynamicRadius=1.0, includeAngular=bool(ang),
                     lanczos_callback=lambda i, err: None)
        return h

    s = handle(order[0])
    for nper in order:
        s.setParameters("advise", N // nper, nper, wallHeight=0.0 if wall else None)
        s.setPositions(p)
        U, W = s.Mdot(F, T)
        Uo, Wo = oracle.mdot(p, F, T, a=1.0, viscosity=1.0, wall=wall, include_angular=ang,
                             nper_batch=nper)
        assert rel_err(U, Uo) <= TOL[precision], nper
        if ang:
            assert rel_err(W, Wo) <= TOL[precision], nper
        fresh = handle(nper)
        fresh.setPositions(p)
        got, want = s.sqrtMdotW_noise(dW), fresh.sqrtMdotW_noise(dW)
        assert got[2] == want[2], nper
        for x, y in zip(got[:2], want[:2]):
            assert (x is None and y is None) or np.array_equal(x, y), nper
