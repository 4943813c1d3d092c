"""The unordered-pair product (csrc/mdot_pairs.cu) on the GPU, against the FP64
oracle at the sizes where its tiles, ranges and passes change, with the
tolerances of every Mdot test: 1e-5 (FP32) and 1e-12 (FP64) relative.
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
    lib.lmg_internal_pairs_max_part(0)


# (N, nper, warps, scratch elements): ragged tiles and slots, batches, ranges cut
# at many steps, several passes of whole batches and of bands of rows
SHAPES = [(1, 1, 0, 0), (2, 1, 0, 0), (33, 11, 0, 0), (63, 63, 0, 0), (65, 65, 1, 0),
          (129, 43, 3, 0), (640, 128, 0, 0), (1537, 1537, 0, 0), (1537, 1537, 37, 0),
          (1537, 1537, 40, 100000), (1998, 333, 16, 60000),
          # many tiles with few partials each: one warp folds a component of a tile
          (9990, 333, 0, 0), (6000, 60, 0, 0), (9990, 333, 300, 300000),
          # tiles with fewer slots in use (17 to 31, and ranges that cut them anywhere)
          (9750, 65, 0, 0), (10000, 100, 0, 0), (8800, 200, 501, 0), (12000, 30, 0, 0)]


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("N,nper,warps,part", SHAPES)
def test_matches_oracle(lib, oracle, precision, wall, N, nper, warps, part):
    """Overlapping, coincident and (above a wall) damped particles included."""
    rng = np.random.default_rng(77 + N + wall)
    p = rng.uniform(0, (N * 4 * np.pi / 3 / 0.15) ** (1 / 3), (N, 3))
    if wall:
        p[:, 2] = rng.uniform(0.3, 9, N)
    if nper > 10:
        p[3] = p[7]
        p[nper - 1] = p[0]
    F, T = rng.normal(size=(2, N, 3))
    assert lib.lmg_internal_sym_override(0, warps) == 0
    assert lib.lmg_internal_pairs_max_part(part) == 0
    p, F, T = (x.astype(np.float32 if precision == "float" else np.float64) for x in (p, F, T))
    for ang, f, t in ((0, F, None), (1, F, T), (1, None, T), (1, F, None)):
        s = make_solver(wall, ang, 1.1, 0.9, precision, N, nper)
        s.setPositions(p)
        U, W = s.Mdot(f, t)
        U2, W2 = s.Mdot(f, t)
        Uo, Wo = oracle.mdot(p, f, t, a=1.1, viscosity=0.9, wall=wall, include_angular=ang,
                             nper_batch=nper)
        assert rel_err(U, Uo) <= TOL[precision], (ang, f is None, t is None)
        assert np.array_equal(U, U2)  # the order of every sum is fixed
        if ang:
            assert rel_err(W, Wo) <= TOL[precision], (f is None, t is None)
            assert np.array_equal(W, W2)


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("N,warm", [(100, False), (100, True), (3000, True)])
def test_captured(lib, precision, N, warm):
    """Mdot in a CUDA graph: after a first call, and for a small system without one
    (nothing can be allocated then: another kernel that needs no scratch)."""
    import torch
    rng = np.random.default_rng(N)
    dt = torch.float32 if precision == "float" else torch.float64
    p = rng.uniform(0, (N * 4 * np.pi / 3 / 0.15) ** (1 / 3), (N, 3)) + 0.5
    p, F, T = (torch.tensor(x, dtype=dt, device="cuda")
               for x in (p, rng.normal(size=(N, 3)), rng.normal(size=(N, 3))))
    s = make_solver(1, 1, 1.0, 1.0, precision, N, N)
    s.setPositions(p)
    if warm:
        s.Mdot(F, T)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        U, W = s.Mdot(F, T)
    F2 = F.clone()
    F.copy_(T)  # read at replay
    g.replay()
    torch.cuda.synchronize()
    got = U.cpu().numpy(), W.cpu().numpy()
    U, W = s.Mdot(T, T)
    assert rel_err(got[0], U.cpu().numpy()) <= TOL[precision]
    assert rel_err(got[1], W.cpu().numpy()) <= TOL[precision]
    F.copy_(F2)


def test_first_call_with_large_tables(lib, oracle):
    """The first product of a plan, whose tables (0.2 MB here) go to the device from
    host memory that has to last until they are there; host memory of that size is
    taken and overwritten at once."""
    nper, nb = 30, 50000
    rng = np.random.default_rng(3)
    p = rng.uniform(0, 12, (nper * nb, 3)).astype(np.float32)
    F, T = rng.normal(size=(2, nper * nb, 3)).astype(np.float32)
    assert lib.lmg_internal_sym_override(0, 1300) == 0
    s = make_solver(1, 1, 1.1, 0.9, "float", nper * nb, nper)
    import torch
    dp, dF, dT = (torch.tensor(x, device="cuda") for x in (p, F, T))
    s.setPositions(dp)
    torch.cuda.synchronize()
    U, W = s.Mdot(dF, dT)
    junk = [np.full(150000 + 1000 * k, -1, np.int64) for k in range(20)]
    U, W = U.cpu().numpy(), W.cpu().numpy()
    assert len(junk) == 20
    some = slice(0, 200 * nper), slice((nb - 200) * nper, nb * nper)
    for sl in some:
        Uo, Wo = oracle.mdot(p[sl], F[sl], T[sl], a=1.1, viscosity=0.9, wall=1, include_angular=1,
                             nper_batch=nper)
        assert rel_err(U[sl], Uo) <= TOL["float"] and rel_err(W[sl], Wo) <= TOL["float"]


@pytest.mark.parametrize("refused", [1, 2])  # its scratch, its cooperative launch
@pytest.mark.parametrize("precision,wall,ang,N", [("float", 0, 1, 900), ("float", 1, 1, 300),
                                                  ("float", 1, 0, 3000), ("double", 1, 1, 500),
                                                  ("double", 0, 0, 700)])
def test_refused(lib, refused, precision, wall, ang, N):
    """Without memory for the partial sums, or where the grid cannot be resident at
    once, the product is mdot_kernel's, bit for bit."""
    rng = np.random.default_rng(N)
    dt = np.float32 if precision == "float" else np.float64
    p = rng.uniform(0.5, 0.5 + (N * 4 * np.pi / 3 / 0.1) ** (1 / 3), (N, 3)).astype(dt)
    F, T = rng.normal(size=(2, N, 3)).astype(dt)
    T = T if ang else None

    def product(s):
        return [x for x in s.Mdot(F, T) if x is not None]

    fresh = lambda: make_solver(wall, ang, 1.0, 1.0, precision)  # noqa: E731
    s, t = fresh(), fresh()
    s.setPositions(p), t.setPositions(p)
    pairs = product(t)
    assert lib.lmg_internal_sym_override(1, 0) == 0
    want = product(s)
    assert lib.lmg_internal_sym_override(0, 0) == 0
    try:
        assert lib.lmg_internal_pairs_refuse(refused) == 0
        for _ in range(2):
            got = product(s)
            assert all(np.array_equal(x, y) for x, y in zip(got, want))
    finally:
        lib.lmg_internal_pairs_refuse(0)
    # memory may be there the next time
    got = product(s)
    assert all(np.array_equal(x, y) for x, y in zip(got, pairs if refused == 1 else want))
    assert not all(np.array_equal(x, y) for x, y in zip(pairs, want))


@pytest.mark.parametrize("far", [1e17, 3e18, 1e19, 1e20, 1e30])
@pytest.mark.parametrize("ang", [0, 1])
def test_particles_far_above_a_wall(lib, oracle, ang, far):
    """Particles put out of the way (padding of uneven batches), up to where the
    product of two heights overflows in FP32: finite and right for all, two of them
    above each other and two in one place included."""
    N = 130
    rng = np.random.default_rng(12)
    p = rng.uniform(1, 12, (N, 3))
    p[100:, 2] = far * rng.uniform(1, 3, 30)
    p[100:110, :2] += far
    p[121, :2] = p[120, :2]
    p[123] = p[122]
    F, T = rng.normal(size=(2, N, 3))
    p, F, T = (x.astype(np.float32) for x in (p, F, T))
    T = T if ang else None
    s = make_solver(1, ang, 1.1, 0.9, "float")
    s.setPositions(p)
    U, W = s.Mdot(F, T)
    # with 64-bit positions nothing overflows
    Uo, Wo = oracle.mdot(p.astype(np.float64), F, T, a=1.1, viscosity=0.9, wall=1,
                         include_angular=ang)
    assert rel_err(U, Uo) <= TOL["float"]
    if ang:
        assert rel_err(W, Wo) <= TOL["float"]


def test_passes_of_whole_batches_carry_nothing(lib):
    """Sums are carried from pass to pass (61 MB here) only where a batch takes
    several passes; these passes hold whole batches, with 4 MB of partial sums."""
    import torch
    nper, nb = 30, 20000
    rng = np.random.default_rng(3)
    p, F, T = (torch.tensor(x, dtype=torch.float32, device="cuda")
               for x in (rng.uniform(1, 12, (nper * nb, 3)), *rng.normal(size=(2, nper * nb, 3))))
    assert lib.lmg_internal_pairs_max_part(1000000) == 0
    s = make_solver(1, 1, 1.1, 0.9, "float", nper * nb, nper)
    s.setPositions(p)
    out = s.Mdot(F, T)
    del out  # (in torch's pool)
    s.clean()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    U, W = s.Mdot(F, T)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 40 << 20


@pytest.mark.parametrize("wall,ang", [(1, 1), (0, 0)])  # the pairs and the symmetric kernel
def test_plans_are_bounded(lib, oracle, wall, ang):
    """A handle whose particles change in number at every call keeps a bounded number
    of plans with device memory, those of captured calls among them."""
    import torch
    rng = np.random.default_rng(8)
    top = 3000
    p, F = (torch.tensor(x, dtype=torch.float32, device="cuda")
            for x in (rng.uniform(1, 60, (top, 3)), rng.normal(size=(top, 3))))
    s = make_solver(wall, ang, 1.1, 0.9, "float")

    def product(n):
        s.setPositions(p[:n])
        return s.Mdot(F[:n])

    first = [x.clone() for x in product(1000) if x is not None]
    for _ in range(2):  # both position buffers at their largest: the graph names one
        product(top)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    s.setPositions(p[:1000])
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        out = [x for x in s.Mdot(F[:1000]) if x is not None]
    used = []
    for k in range(4):
        for n in range(1500 + 100 * k, 1600 + 100 * k):
            product(n)
        torch.cuda.synchronize()
        used.append(torch.cuda.mem_get_info()[0])
    # 100 further plans take nothing (2 MB: the unit in which memory is given out)
    assert used[1] - used[3] <= 2 << 20, used
    for _ in range(2):
        s.setPositions(p[:1000])
    torch.cuda.synchronize()
    for x in out:
        x.zero_()
    g.replay()
    torch.cuda.synchronize()
    for x, y in zip(out, first):
        assert torch.equal(x, y)
