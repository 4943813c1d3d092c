"""Host plan of the unordered-pair product (no GPU needed).

lmg_internal_pairs_plan builds the passes, the step ranges and the
lists of cut tile pairs; these tests walk them as the kernel does
(csrc/mdot_pairs.cu) and check that every rotation step of every tile pair is
taken once, that every partial the fold reads was written in the same pass (and
once), inside the scratch, that the fold reads every partial that was written,
and that the carried sums open and close once per batch.
"""
import ctypes

import numpy as np
import pytest


@pytest.fixture(scope="module")
def lib():
    from libmobility_gb300 import _capi
    return _capi.load()


def plan(lib, N, nper, ang, double, resident, warps, max_part):
    info = np.zeros(6, np.int64)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    args = (N, nper, ang, double, resident, warps, max_part, ptr(info))
    assert lib.lmg_internal_pairs_plan(*args, None, None) == 0
    passes = np.zeros((int(info[0]), 7), np.int64)
    cuts = np.zeros(int(info[1]), np.int32)
    assert lib.lmg_internal_pairs_plan(*args, ptr(passes), ptr(cuts)) == 0
    return passes, cuts, int(info[2]), int(info[3]), int(info[4]), int(info[5])


def before(tpb, r):
    b, i = divmod(r, tpb)
    return b * (tpb * (tpb + 1) // 2) + i * tpb - i * (i - 1) // 2


@pytest.mark.parametrize("N,nper,warps,max_part", [
    (1, 1, 0, 0), (64, 64, 0, 0), (65, 65, 1, 0), (333 * 7, 333, 0, 0), (2048, 2048, 0, 0),
    (2048, 2048, 37, 0), (20 * 100, 20, 0, 0), (4096, 4096, 5, 0),
    (2048, 2048, 40, 40000), (1000 * 3, 1000, 30, 40000), (300 * 8, 300, 16, 9000)])
@pytest.mark.parametrize("double", [0, 1])
@pytest.mark.parametrize("ang", [0, 1])
def test_every_step_and_partial_once(lib, N, nper, warps, max_part, double, ang):
    tile = 32 if double else 64
    el = (6 if ang else 3) * tile
    # under a scratch limit only a few blocks are resident: two slots a warp
    resident = 3 if max_part else 152 * 3
    passes, cuts, part, acc, tpb, S = plan(lib, N, nper, ang, double, resident, warps, max_part)
    nb = N // nper
    rows = nb * tpb
    assert tpb == -(-nper // tile)
    # equal tiles of S slots hold a batch; with work for every warp no slot more
    # than needed, otherwise whole tiles
    ns = 1 if double else 2
    assert 1 <= S <= 32 and tpb * S * ns >= nper and (tpb - 1) * S * ns < nper
    if 32 * nb * tpb * (tpb + 1) // 2 > 4 * 4 * resident:
        assert tpb * (S - 1) * ns < nper
    else:
        assert S == 32
    assert passes[0, 0] == 0 and passes[-1, 1] == rows
    assert np.array_equal(passes[1:, 0], passes[:-1, 1])
    assert (acc > 0) == (len(passes) > 1)
    if acc:
        assert acc == 2 * rows * el
    if max_part:
        assert len(passes) > 1
    for row0, row1, steps, per_warp, nwarps, grid, off in passes.tolist():
        # whole batches, or a band of one
        assert row0 % tpb == 0 or row1 <= (row0 // tpb + 1) * tpb
        assert row1 % tpb == 0 or row1 - row0 < tpb
        P0 = before(tpb, row0)
        npairs = before(tpb, row1) - P0
        assert steps == S * npairs and nwarps <= 4 * grid and grid <= resident
        assert (nwarps - 1) * per_warp < steps <= nwarps * per_warp
        slot_row, slot_irow = npairs, npairs + row1 - row0
        slot_cut = slot_irow + nwarps
        assert (slot_cut + nwarps) * el <= part
        taken = np.zeros(steps, np.int8)
        written = {}  # slot -> tile its sums belong to
        pairs = [(r, J) for r in range(row0, row1) for J in range(r, (r // tpb + 1) * tpb)]
        assert len(pairs) == npairs
        for w in range(nwarps):
            x, left = w * per_warp, min(per_warp, steps - w * per_warp)
            new_pair = x % S == 0
            new_row = new_pair and pairs[x // S][0] == pairs[x // S][1]
            while left > 0:
                p, k = x // S, x % S
                r, J = pairs[p]
                n = min(S - k, left)
                taken[x:x + n] += 1
                if r != J:
                    slot = p if new_pair else slot_cut + w
                    assert slot not in written
                    written[slot] = J
                x, left, new_pair = x + n, left - n, True
                if p + 1 == npairs or pairs[p + 1][0] != r or left == 0:
                    slot = slot_row + r - row0 if new_row else slot_irow + w
                    assert slot not in written
                    written[slot] = r
                    new_row = True
        assert (taken == 1).all()
        # the fold
        begin = cuts[off:off + rows + 1]
        cut_warps = cuts[off + rows + 1:]
        read = {}
        for t in range(row0 // tpb * tpb, ((row1 - 1) // tpb + 1) * tpb):
            b0 = t // tpb * tpb
            for r in range(max(b0, row0), min(t, row1)):
                I = r - b0
                slot = before(tpb, b0) - P0 + I * tpb - I * (I - 1) // 2 + t - r
                read[slot] = t
            if row0 <= t < row1:
                xs, xe = S * (before(tpb, t) - P0), S * (before(tpb, t + 1) - P0)
                read[slot_row + t - row0] = t
                for g in range(xs // per_warp + 1, (xe - 1) // per_warp + 1):
                    read[slot_irow + g] = t
            for g in cut_warps[begin[t]:begin[t + 1]]:
                read[slot_cut + int(g)] = t
        assert read == written


@pytest.mark.parametrize("S", [1, 2, 17, 31, 32])
def test_rotation_steps_cover_a_tile_pair(S):
    """Lane l's slot meets slot (l + k) mod S at step k: every pair of slots
    once over the S steps, and no slot twice in a step; the lanes past S keep to
    their own.  The slots of a lane's flagged steps, as a mask: bit k moves to
    (k + l) mod S."""
    lane = np.arange(32)
    seen = np.zeros((S, S), int)
    for k in range(S):
        s = np.where(lane >= S, lane, np.where(lane + k >= S, lane + k - S, lane + k))
        assert len(set(s)) == 32
        seen[lane[:S], s[:S]] += 1
        for l in range(S):
            at = (1 << k) << l
            assert ((at | (at >> S)) & ((1 << S) - 1)) == 1 << s[l]
    assert (seen == 1).all()
