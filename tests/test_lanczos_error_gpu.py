"""The error a convergence check reports, |y_i - y_(i-1)| / |y_(i-1)|, against the
same in 64 bits from the two iterates themselves.

Iterates do not depend on the tolerance, so one just above a reported error
returns the iterate of that check (prefactor 1, added to zeros: exact).

Bound, with u = 2^-53: a value's square is rounded once (differences of FP32 values
are exact) and then meets at most A additions that round, A = 9 for 300 values (3
levels over the eight values of a warp, 3 over the block's warps, 3 over the five
blocks), 16 for more (2 of a thread's own, 6, 3 partials of a thread, 8 - 3 over
the last block); a square root halves that and rounds, as does the quotient:
((A + 1) / 2 + 1) 2 + 1 units for both, and one for the sums here.
"""
import math

import numpy as np
import pytest

from test_mdot_gpu import make_solver

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("wall,ang,N,adds,seeds", [(1, 0, 100, 9, 24), (0, 0, 999, 16, 3),
                                                   (1, 1, 500, 16, 3), (0, 0, 22000, 16, 1)])
def test_error_in_64_bits(cuda, wall, ang, N, adds, seeds):
    """Vectors of up to 65536 values take four threads a value, longer ones one."""
    worst = 0.0
    for seed in range(seeds):
        rng = np.random.default_rng(N + 1000 * seed)
        p = rng.uniform(0.6, 0.6 + (N * 4 * np.pi / 3 / 0.05) ** (1 / 3), (N, 3))
        dW = rng.normal(size=N * (6 if ang else 3))
        errs = {}

        def solve(tol):
            s = make_solver(wall, ang, 1.0, 1.0, "float")
            s.initialize(viscosity=1.0, hydrodynamicRadius=1.0, includeAngular=bool(ang),
                         tolerance=tol, lanczos_callback=lambda i, e: errs.__setitem__(i, e))
            s.setPositions(p)
            u, w, it, res = s.sqrtMdotW_noise(dW)
            y = np.concatenate([np.asarray(x, np.float64).ravel() for x in (u, w)
                                if x is not None])
            return y, it, res

        _, last, _ = solve(1e-4)
        seen = dict(errs)
        for i in range(max(3, last - 5), last + 1):
            before, it0, _ = solve(seen[i - 1] * (1 + 1e-9))
            now, it1, res = solve(seen[i] * (1 + 1e-9))
            if (it0, it1) != (i - 1, i):
                continue  # the error did not fall at this step
            want = math.sqrt(math.fsum((now - before) ** 2) / math.fsum(before ** 2))
            worst = max(worst, abs(res / want - 1))
    assert worst <= (adds + 1 + 2 + 1 + 1) * U
