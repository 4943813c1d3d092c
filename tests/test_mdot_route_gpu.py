"""Products on both sides of the lines between the kernels (csrc/mdot_route.hpp),
against the FP64 oracle with the tolerances of every Mdot, 1e-5 (FP32) and 1e-12
(FP64) relative; and the unordered-pair kernel at the sizes that the rule gives
to another one (capping its warps, here at far more than there are, selects it).
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


# batches x particles: a handful, tiny batches below and above the lines, whole
# warps and tiles, and batches the symmetric kernel takes or leaves
SIZES = [(1, 1), (1, 2), (1, 3), (1, 9), (1, 16), (1, 17), (1, 24), (1, 25), (4, 4), (152, 2),
         (153, 2), (400, 3), (1216, 16), (1217, 12), (400, 8), (700, 16), (304, 32), (200, 64),
         (160, 128), (20, 256), (40, 256), (80, 96), (77, 100), (1300, 24), (3000, 1)]


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("forced", [0, 1000000])
@pytest.mark.parametrize("nb,nper", SIZES)
def test_matches_oracle(lib, oracle, precision, wall, forced, nb, nper):
    N = nb * nper
    rng = np.random.default_rng(31 + N + wall)
    p = rng.uniform(0, (nper * 4 * np.pi / 3 / 0.15) ** (1 / 3) + 1, (N, 3))
    if wall:
        p[:, 2] = rng.uniform(0.3, 9, N)
    if nper > 10:
        p[3] = p[7]
    F, T = rng.normal(size=(2, N, 3))
    p, F, T = (x.astype(np.float32 if precision == "float" else np.float64) for x in (p, F, T))
    assert lib.lmg_internal_sym_override(0, forced) == 0
    for ang, f, t in ((0, F, None), (1, F, T), (1, None, T), (1, F, None)):
        s = make_solver(wall, ang, 1.1, 0.9, precision, N, nper)
        s.setPositions(p)
        U, W = s.Mdot(f, t)
        Uo, Wo = oracle.mdot(p, f, t, a=1.1, viscosity=0.9, wall=wall, include_angular=ang,
                             nper_batch=nper)
        assert rel_err(U, Uo) <= TOL[precision], (ang, f is None, t is None)
        if ang:
            assert rel_err(W, Wo) <= TOL[precision], (f is None, t is None)
