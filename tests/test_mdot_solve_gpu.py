"""The products of a solve (mdot_kernel, csrc/mdot.cuh) on the GPU against the
FP64 oracle, at the sizes where its launch changes: ragged source tiles, former
splits of several tiles cut into one tile each, close wall pairs dealt out
(up to 4096 sources) or met in place, more close pairs than the list of a warp
holds, batches whose tiles cover two.  Tolerances of every Mdot test, 1e-5
(FP32) and 1e-12 (FP64) relative.
"""
import numpy as np
import pytest

from test_mdot_gpu import make_solver, rel_err

pytestmark = pytest.mark.gpu
TOL = {"float": 1e-5, "double": 1e-12}


@pytest.fixture()
def tiled(cuda):
    from libmobility_gb300 import _capi
    lib = _capi.load()
    assert lib.lmg_internal_sym_override(1, 0) == 0  # mdot_kernel for every product
    yield lib
    lib.lmg_internal_sym_override(0, 0)


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("N,nper,dense", [(1, 1, 1), (33, 33, 1), (127, 127, 8), (129, 129, 1),
                                          (300, 300, 1), (512, 512, 30), (999, 333, 1),
                                          (1000, 1000, 1), (2000, 2000, 1), (4225, 4225, 1)])
def test_matches_oracle(tiled, oracle, precision, wall, N, nper, dense):
    """`dense` times the particles per volume of the others (30: a target has
    dozens of overlapping sources in every tile)."""
    if precision == "double" and N > 2000:
        pytest.skip("the launch is the one of N = 2000")
    rng = np.random.default_rng(5 + N + wall)
    side = (N * 4 * np.pi / 3 / (0.1 * dense)) ** (1 / 3)
    p = rng.uniform(0, side, (N, 3))
    if wall:
        p[:, 2] += 0.4
    if nper > 8:
        p[3] = p[6]
    F, T = rng.normal(size=(2, N, 3))
    p, F, T = (x.astype(np.float32 if precision == "float" else np.float64) for x in (p, F, T))
    for ang, f, t in ((0, F, None), (1, F, T)):
        s = make_solver(wall, ang, 1.0, 1.0, precision, N, nper)
        s.setPositions(p)
        U, W = s.Mdot(f, t)
        Uo, Wo = oracle.mdot(p, f, t, a=1.0, viscosity=1.0, wall=wall, include_angular=ang,
                             nper_batch=nper)
        assert rel_err(U, Uo) <= TOL[precision], ang
        if ang:
            assert rel_err(W, Wo) <= TOL[precision]


@pytest.mark.parametrize("N", [5000, 16384, 33001, 70000])
def test_symmetric_fold(cuda, N):
    """The symmetric product's fold with 8, 16 and 32 shares an element (one, two
    and four turns of 8 lanes) and more slots than one pass over them, against
    the FP64 product of the same (single precision) inputs."""
    rng = np.random.default_rng(N)
    p = rng.uniform(0, (N * 4 * np.pi / 3 / 0.1) ** (1 / 3), (N, 3)).astype(np.float32)
    F = rng.normal(size=(N, 3)).astype(np.float32)
    out = {}
    for precision, dtype in (("float", np.float32), ("double", np.float64)):
        s = make_solver(0, 0, 1.0, 1.0, precision, N, N)
        s.setPositions(p.astype(dtype))
        out[precision] = s.Mdot(F.astype(dtype))[0]
    assert rel_err(out["float"], out["double"]) <= TOL["float"]


@pytest.mark.parametrize("power", [60, 100])
@pytest.mark.parametrize("N", [200, 3000])
def test_large_noise(cuda, N, power):
    """The convergence check sums FP32 squares at a scale of its own, so noise whose
    squares are out of range stops at the same iteration, and the result is that
    of ordinary noise times the same power of two, bit for bit.  (Not for small
    noise: the recurrence takes beta < 1e-3 alpha / |z| for a breakdown, as the
    reference does, LanczosAlgorithm.cu:144, and ends early below |z| of about
    0.01.)"""
    rng = np.random.default_rng(N)
    p = rng.uniform(0, (N * 4 * np.pi / 3 / 0.1) ** (1 / 3), (N, 3)).astype(np.float32)
    z = rng.normal(size=(N, 3)).astype(np.float32)
    out = []
    for scale in (0, power):
        s = make_solver(0, 0, 1.0, 1.0, "float", N, N)
        s.setPositions(p)
        y, _, iterations, _ = s.sqrtMdotW_noise(np.ldexp(z, scale).astype(np.float32))
        out.append((np.asarray(y), iterations))
    assert out[0][1] == out[1][1]
    assert np.array_equal(np.ldexp(out[0][0], power).astype(np.float32), out[1][0])
