"""A grid barrier whose wait runs out (here: after no polls) in the symmetric and the
unordered-pair product: every sum folded behind it is NaN, never memory that
nobody wrote; the call that waits for its result raises the error, an asynchronous
one leaves it to the next product or synchronize; and the handle then works on.
"""
import numpy as np
import pytest

from test_mdot_gpu import make_solver, rel_err

pytestmark = pytest.mark.gpu
TOL = {"float": 1e-5, "double": 1e-12}
TIMEOUT = 7  # LMG_ERR_TIMEOUT


@pytest.fixture()
def lib(cuda):
    from libmobility_gb300 import _capi
    lib = _capi.load()
    yield lib
    lib.lmg_internal_barrier_spins(-1)
    lib.lmg_internal_pairs_max_part(0)


def system(N, ang, precision):
    rng = np.random.default_rng(N)
    dt = np.float32 if precision == "float" else np.float64
    p = rng.uniform(0.5, 0.5 + (N * 4 * np.pi / 3 / 0.1) ** (1 / 3), (N, 3)).astype(dt)
    F, T = rng.normal(size=(2, N, 3)).astype(dt)
    return p, F, T if ang else None


# the symmetric kernel; the pairs; the same in several passes
CASES = [("float", 0, 0, 2000, 0), ("float", 0, 1, 700, 0), ("float", 1, 1, 300, 0),
         ("double", 1, 0, 400, 0), ("float", 1, 0, 1500, 60000)]


@pytest.mark.parametrize("precision,wall,ang,N,part", CASES)
def test_a_wait_that_runs_out(lib, oracle, precision, wall, ang, N, part):
    import torch
    assert lib.lmg_internal_pairs_max_part(part) == 0
    p, F, T = system(N, ang, precision)
    dp, dF = torch.tensor(p, device="cuda"), torch.tensor(F, device="cuda")
    dT = None if T is None else torch.tensor(T, device="cuda")
    Uo, Wo = oracle.mdot(p, F, T, a=1.0, viscosity=1.0, wall=wall, include_angular=ang)
    s = make_solver(wall, ang, 1.0, 1.0, precision)
    s.setPositions(dp)

    def right():
        U, W = s.Mdot(dF, dT)
        assert lib.lmg_synchronize(s._h) == 0
        assert rel_err(U.cpu().numpy(), Uo) <= TOL[precision]
        if ang:
            assert rel_err(W.cpu().numpy(), Wo) <= TOL[precision]

    right()
    # device arrays: synchronize raises it, once
    lib.lmg_internal_barrier_spins(0)
    U, W = s.Mdot(dF, dT)
    torch.cuda.synchronize()
    lib.lmg_internal_barrier_spins(-1)
    assert torch.isnan(U).all() and (W is None or torch.isnan(W).all())
    assert lib.lmg_synchronize(s._h) == TIMEOUT
    assert b"timed out" in lib.lmg_last_error(s._h)
    right()
    # or the next product
    lib.lmg_internal_barrier_spins(0)
    s.Mdot(dF, dT)
    torch.cuda.synchronize()
    lib.lmg_internal_barrier_spins(-1)
    with pytest.raises(RuntimeError, match="timed out"):
        s.Mdot(dF, dT)
    right()
    # host arrays: the call itself
    lib.lmg_internal_barrier_spins(0)
    with pytest.raises(RuntimeError, match="timed out"):
        s.Mdot(F, T)
    if wall:
        with pytest.raises(RuntimeError, match="timed out"):
            s.setPositions(p)
            s.divM(1.0)
        s.setPositions(dp)
    lib.lmg_internal_barrier_spins(-1)
    right()


def test_in_a_solve(lib):
    """A solve with the symmetric product raises it, and the next one is right."""
    p, F, _ = system(1500, 0, "float")
    s = make_solver(0, 0, 1.0, 1.0, "float")
    s.setPositions(p)
    dW = F.ravel()
    want = s.sqrtMdotW_noise(dW)
    lib.lmg_internal_barrier_spins(0)
    with pytest.raises(RuntimeError, match="timed out"):
        s.sqrtMdotW_noise(dW)
    lib.lmg_internal_barrier_spins(-1)
    got = s.sqrtMdotW_noise(dW)
    assert np.linalg.norm(got[0] - want[0]) <= 1e-3 * np.linalg.norm(want[0])
