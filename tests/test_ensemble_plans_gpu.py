"""Launch plans of the ensemble's autotuner: every plan it may pick gives every
system the whole sum over its sources.

Systems whose padded size is an odd multiple of 128 lie side by side in a
group, so a tile of 256 targets (two per thread) would cover two of them and
need the sources of both; the splits are made for one.  Products against the
FP64 oracle, 1e-5 relative as every FP32 Mdot, on fresh handles, since the
choice is made by timing.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("repeat", range(4))
@pytest.mark.parametrize("sizes", [[300, 310, 290, 380, 330, 350], [100, 90, 120, 70],
                                   [600, 700, 620, 760], [200, 256, 250, 130, 140]])
def test_tuned_plans_sum_every_source(cuda, oracle, sizes, repeat):
    from libmobility_gb300.ensemble import Ensemble
    rng = np.random.default_rng(repeat + sum(sizes))
    sizes = sizes * 4
    geometry = ["open" if k % 2 else "single_wall" for k in range(len(sizes))]
    pos = [np.column_stack([rng.uniform(0, n ** 0.5, (n, 2)), rng.uniform(1.5, 20, n)])
           for n in sizes]
    F = [rng.normal(size=(n, 3)) for n in sizes]
    e = Ensemble(precision="float")
    e.setSystems(sizes, geometry, [0.0] * len(sizes))
    e.initialize(1.0, 1.0, tolerance=1e-4, seed=1)
    e.setPositions(np.concatenate(pos).astype(np.float32))
    U = e.Mdot(np.concatenate(F).astype(np.float32))
    b = 0
    for p, f, g in zip(pos, F, geometry):
        Uo, _ = oracle.mdot(p.astype(np.float32), f.astype(np.float32), None, a=1.0,
                            viscosity=1.0, wall=g != "open", include_angular=0)
        assert np.abs(U[b:b + len(p)] - Uo).max() <= 1e-5 * np.abs(Uo).max(), (len(p), g)
        b += len(p)


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("sizes", [[1, 2, 100, 341], [341, 342, 500], [300, 700, 1365, 1366],
                                   [2049, 2730, 60]])
def test_one_launch_step_is_the_three_kernel_step(cuda, sizes, precision):
    """Systems of up to 8 chunks of 1024 values take one cluster launch a step.
    With one larger system beside them (4100 particles, its own group, so the
    others' products stay the same) the step goes through three kernels: same
    arithmetic in the same order, so the same bits."""
    from libmobility_gb300.ensemble import Ensemble
    rng = np.random.default_rng(sum(sizes))
    sizes = sizes + [4100]
    pos = np.concatenate([rng.uniform(0, 2.5 * n ** (1 / 3), (n, 3)) for n in sizes])
    dW = rng.normal(size=(sum(sizes), 3))
    dtype = np.float32 if precision == "float" else np.float64
    out = []
    for k in (len(sizes) - 1, len(sizes)):
        m = sum(sizes[:k])
        e = Ensemble(precision=precision)
        e.setSystems(sizes[:k], ["open"] * k, [0.0] * k)
        e.initialize(1.0, 1.0, tolerance=1e-4, seed=1, autotune=False)
        e.setPositions(pos[:m].astype(dtype))
        r = e.sqrtMdotW(dW[:m].astype(dtype))
        out.append((np.asarray(r[0]), np.asarray(r[1])))
    m = sum(sizes[:-1])
    assert (out[0][1] == out[1][1][:-1]).all()
    assert np.array_equal(out[0][0][:m], out[1][0][:m])


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("sizes,wide", [([300, 310, 290, 380], False), ([200, 256, 250, 140], True),
                                        ([600, 700, 620, 760], False), ([400, 512, 390, 400], None),
                                        ([500, 400, 510, 390], True), ([300], True),
                                        ([800, 900, 1000, 990], False)])
def test_tuner_tries_wide_tiles_only_within_systems(cuda, sizes, wide, precision):
    """Whatever the timing says: tiles of two targets a thread are among the plans
    tried only where none covers two systems, that is where every system but the
    last of its group is padded to a multiple of 256."""
    from libmobility_gb300.ensemble import Ensemble
    rng = np.random.default_rng(0)
    e = Ensemble(precision=precision)
    e.setSystems(sizes, ["open"] * len(sizes), [0.0] * len(sizes))
    e.initialize(1.0, 1.0, tolerance=1e-4, seed=1)
    n = sum(sizes)
    dtype = np.float32 if precision == "float" else np.float64
    e.setPositions(rng.uniform(0, 40, (n, 3)).astype(dtype))
    e.Mdot(rng.normal(size=(n, 3)).astype(dtype))
    groups = e.describe()["groups"]
    bucket = lambda s: s.bit_length() - 1  # noqa: E731
    assert len(groups) == len({bucket(s) for s in sizes})
    for g in groups:
        lo, hi = g["size_range"]
        padded = [-(-s // 128) * 128 for s in sizes if lo <= s <= hi]
        tried = {t for t, _, _ in g["trials_ms"]}
        within = all(p % 256 == 0 for p in padded[:-1])
        assert tried == ({1, 2} if within else {1})
        if wide is not None:
            assert within == wide
