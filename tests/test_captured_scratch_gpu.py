"""A captured product goes on being right while other calls of its handle, on the same
positions, make its scratch grow: the graph keeps the allocation that it names.
"""
import numpy as np
import pytest

from test_mdot_gpu import make_solver

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib(cuda):
    from libmobility_gb300 import _capi
    lib = _capi.load()
    yield lib
    lib.lmg_internal_mdot_plan_override(0, 0)
    lib.lmg_internal_sym_override(0, 0)


# mdot_kernel by the rule (forces alone with angular velocities in open space, tiny
# batches) and the pairs
@pytest.mark.parametrize("wall,ang,N,nper,torques", [(0, 1, 6000, 6000, False),
                                                     (1, 1, 6000, 5, True),
                                                     (1, 1, 2000, 2000, True)])
def test_scratch_grows_under_a_graph(lib, wall, ang, N, nper, torques):
    import torch
    rng = np.random.default_rng(N)
    p, F, T = (torch.tensor(x, dtype=torch.float32, device="cuda")
               for x in (rng.uniform(1, 60, (N, 3)), *rng.normal(size=(2, N, 3))))
    s = make_solver(wall, ang, 1.0, 1.0, "float", N, nper)
    s.setPositions(p)
    args = (F, T) if torques else (F,)
    want = [x.clone() for x in s.Mdot(*args)]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = s.Mdot(*args)

    def replayed():
        for x in out:
            x.zero_()
        g.replay()
        torch.cuda.synchronize()
        return all(torch.equal(x, y) for x, y in zip(out, want))

    assert replayed()
    # more splits, so more partial sums, in mdot_kernel; a solve; the same calls again
    for splits in (8, 40, 64):
        assert lib.lmg_internal_mdot_plan_override(1, splits) == 0
        a = s.Mdot(F, T)
        torch.cuda.synchronize()
        assert replayed()
        b = s.Mdot(F, T)
        assert all(torch.equal(x, y) for x, y in zip(a, b))
    assert lib.lmg_internal_mdot_plan_override(0, 0) == 0
    s.sqrtMdotW_noise(torch.cat([F.reshape(-1), T.reshape(-1)]))
    assert replayed()
    junk = [torch.full((1 << 22,), float("nan"), device="cuda") for _ in range(8)]
    assert replayed() and len(junk) == 8
    assert all(torch.equal(x, y) for x, y in zip(s.Mdot(*args), want))
