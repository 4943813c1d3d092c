"""Which kernel a product outside a solve takes (csrc/mdot_route.hpp), at sizes
whose kernels were timed on a GB300: the faster one, by more than the runs of
one side differ, on both sides of every line.
"""
import pytest

TILED, SYMMETRIC, PAIRS = 0, 1, 2
SMS = 152

# (fp64, wall, angular, one of F and T alone, batches, particles of one, kernel)
CASES = [
    # a handful of particles, and from there on
    (0, 0, 0, 0, 1, 1, TILED), (0, 0, 1, 0, 1, 10, TILED), (0, 1, 1, 0, 1, 10, TILED),
    (0, 0, 0, 0, 1, 50, PAIRS), (0, 1, 0, 0, 1, 24, PAIRS), (0, 1, 1, 0, 1, 32, PAIRS),
    (1, 0, 0, 0, 1, 5, TILED), (1, 0, 0, 0, 1, 12, PAIRS), (1, 1, 1, 0, 1, 1, TILED),
    (1, 1, 1, 0, 1, 6, PAIRS),
    # many tiny batches
    (0, 0, 0, 0, 1000, 1, TILED), (0, 0, 1, 0, 500, 2, TILED), (0, 1, 0, 0, 100000, 1, TILED),
    (0, 1, 1, 0, 1000000, 1, TILED), (0, 1, 1, 0, 125000, 8, TILED), (0, 0, 1, 0, 6250, 16, TILED),
    (0, 1, 1, 0, 3125, 32, TILED), (0, 1, 0, 0, 25000, 4, TILED), (0, 0, 0, 0, 250000, 4, TILED),
    (0, 0, 1, 0, 4166, 24, TILED), (0, 0, 1, 0, 800, 128, TILED),
    (0, 1, 1, 0, 150, 2, PAIRS), (0, 1, 0, 0, 625, 16, PAIRS), (0, 0, 1, 0, 300 // 16, 16, PAIRS),
    (0, 1, 1, 0, 5000, 20, PAIRS), (0, 1, 0, 0, 3125, 32, PAIRS), (0, 0, 1, 0, 2000, 50, PAIRS),
    (0, 1, 1, 0, 1562, 64, PAIRS), (0, 0, 0, 0, 64, 333, PAIRS),
    (1, 0, 0, 0, 100000, 1, TILED), (1, 0, 1, 0, 12500, 8, TILED), (1, 0, 0, 0, 6250, 16, TILED),
    (1, 1, 0, 0, 100000, 1, TILED), (1, 1, 1, 0, 100000, 1, TILED), (1, 0, 1, 0, 3125, 32, TILED),
    (1, 0, 0, 0, 300, 4, PAIRS), (1, 0, 0, 0, 5000, 20, PAIRS), (1, 1, 0, 0, 25000, 4, PAIRS),
    (1, 1, 1, 0, 12500, 8, PAIRS), (1, 0, 1, 0, 625, 16, PAIRS),
    # FP32 open forces: tiles of 128
    (0, 0, 0, 0, 1, 4096, SYMMETRIC), (0, 0, 0, 0, 1, 384, SYMMETRIC), (0, 0, 0, 0, 1, 383, PAIRS),
    (0, 0, 0, 0, 78, 256, SYMMETRIC), (0, 0, 0, 0, 234, 96, SYMMETRIC),
    (0, 0, 0, 0, 400, 128, SYMMETRIC), (0, 0, 0, 0, 20, 96, PAIRS), (0, 0, 0, 0, 200, 192, PAIRS),
    (0, 0, 0, 0, 400, 260, PAIRS), (0, 0, 0, 0, 70, 352, SYMMETRIC),
    # forces or torques alone: half the work in mdot_kernel
    (0, 0, 1, 1, 1, 16384, TILED), (0, 0, 1, 1, 1, 3000, PAIRS), (0, 0, 1, 1, 2000, 100, TILED),
    (0, 0, 1, 1, 400, 200, PAIRS), (0, 0, 1, 1, 100, 256, TILED), (0, 0, 1, 1, 100, 500, PAIRS),
    (0, 0, 1, 1, 2000, 20, PAIRS), (0, 1, 1, 1, 1, 16384, PAIRS),
    (0, 0, 1, 1, 4, 2500, PAIRS), (0, 0, 1, 1, 2, 4000, PAIRS), (0, 0, 1, 1, 2, 9001, PAIRS),
    (0, 0, 1, 1, 2, 16384, TILED), (0, 0, 1, 1, 10, 512, TILED), (0, 0, 1, 1, 2000, 72, TILED),
    (0, 0, 1, 1, 267, 160, PAIRS), (0, 0, 1, 1, 1000, 160, TILED),
    (0, 0, 1, 1, 160, 600, PAIRS), (0, 0, 1, 1, 153, 400, PAIRS), (0, 0, 1, 1, 400, 96, TILED),
    (0, 1, 1, 0, 84, 1, TILED), (0, 0, 0, 0, 49, 1, TILED), (1, 1, 0, 0, 6, 1, TILED),
    (0, 0, 1, 0, 117, 1, PAIRS), (0, 1, 0, 0, 95, 1, PAIRS), (0, 0, 1, 0, 30, 1, TILED),
    (0, 0, 1, 1, 1, 28, TILED), (0, 1, 1, 1, 1, 19, TILED), (0, 1, 1, 1, 988, 6, TILED),
    (1, 0, 1, 1, 721, 3, PAIRS), (1, 0, 1, 1, 334, 32, TILED), (1, 0, 1, 1, 1427, 8, TILED), (1, 0, 1, 1, 619, 1, TILED), (1, 0, 1, 1, 1, 9, TILED),
    (1, 1, 0, 0, 300, 1, PAIRS), (0, 0, 0, 0, 2, 17, TILED), (0, 1, 1, 0, 655, 12, PAIRS),
    (0, 1, 1, 0, 322, 7, PAIRS), (0, 0, 1, 0, 375, 8, TILED), (0, 1, 1, 0, 2500, 12, TILED),
    (1, 0, 1, 1, 369, 64, TILED), (1, 0, 1, 1, 2591, 3, TILED), (1, 1, 1, 1, 1, 5, TILED),
    (1, 0, 1, 1, 160, 65, PAIRS), (1, 0, 1, 1, 200, 48, PAIRS), (1, 0, 1, 1, 400, 33, TILED),
    (1, 0, 1, 1, 400, 64, TILED), (1, 0, 1, 1, 100, 200, PAIRS), (1, 0, 1, 1, 1, 4096, PAIRS),
    (1, 1, 1, 1, 400, 64, PAIRS),
    # both: everything larger
    (0, 0, 1, 0, 1, 16384, PAIRS), (0, 1, 1, 0, 1, 16384, PAIRS), (0, 1, 0, 0, 1, 100003, PAIRS),
    (1, 1, 1, 0, 1, 3001, PAIRS), (1, 0, 0, 0, 1, 4096, PAIRS),
]


@pytest.mark.parametrize("fp64,wall,ang,one,nb,nper,kernel", CASES)
def test_route(fp64, wall, ang, one, nb, nper, kernel):
    from libmobility_gb300 import _capi
    lib = _capi.load()
    assert lib.lmg_internal_mdot_route(fp64, wall, ang, one, nb * nper, nper, SMS) == kernel
