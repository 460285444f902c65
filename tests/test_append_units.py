"""The appends kernel's units of massive tiles (csrc/sfp_step.cuh:
sfp_appends_body, sfp_append_tile), restated from their index arithmetic:
every tile with events is in exactly one unit, a unit lies inside one
segment and one super-tile, its particles follow one another and fit the
warp's list, and a unit's first child's rank is the number of events before
it, at tile lengths and populations around the rule's edges."""
import numpy as np
import pytest

SUPER, TILE_MAX, TARGET_M = 64, 1024, 16384


def unit_tiles(n_tiles, n_warps, tile):
    u = 1
    while n_tiles // u > n_warps and tile * u < TILE_MAX and u < SUPER:
        u <<= 1
    return u


@pytest.mark.parametrize("n_warps", [8, 2368, 3552])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 2048, 500_001, 524_288, 524_289, 1_048_577, 16_777_217])
def test_units_cover_every_tile_once(n, n_warps):
    rng = np.random.default_rng(n % 1000 + n_warps)
    parts = sorted(rng.integers(0, n + 1, 2))  # three segments, some empty
    sizes = [parts[0], parts[1] - parts[0], n - parts[1]]
    tile = 32
    while tile < TILE_MAX and tile * TARGET_M < n:
        tile <<= 1
    start, acc = [], 0
    for s in sizes:
        acc = -(-acc // SUPER) * SUPER
        start.append(acc)
        acc += -(-s // tile)
    n_tiles = acc
    u = unit_tiles(n_tiles, n_warps, tile)
    assert SUPER % u == 0 and tile * u <= TILE_MAX
    cnt = np.zeros(n_tiles, dtype=np.int64)
    for a, s in zip(start, sizes):
        k = -(-s // tile)
        cnt[a:a + k] = rng.integers(0, 3, k)
    starts = np.array(start)
    seen = 0
    units = range(-(-n_tiles // u))
    if len(units) > 4000:  # the ends and a sample between
        units = sorted(set(range(50)) | set(range(len(units) - 50, len(units)))
                       | set(int(v) for v in rng.integers(0, len(units), 500)))
    total = np.concatenate([[0], np.cumsum(cnt)])
    for j in units:
        t0, t1 = j * u, min(n_tiles, j * u + u)
        c = int(total[t1] - total[t0])
        seen += c
        if c == 0:
            continue
        assert t0 // SUPER == (t1 - 1) // SUPER
        pos = len(starts) - 1 - int(np.argmax(starts[::-1] <= t0))
        base = (t0 - start[pos]) * tile
        length = min(sizes[pos] - base, tile * u)
        assert 0 < length <= TILE_MAX and base % 32 == 0
        # the unit's tiles with events are its segment's tiles of these particles
        own = range(t0, start[pos] + -(-(base + length) // tile))
        assert int(total[own.stop] - total[own.start]) == c
        first = int(total[(t0 // SUPER) * SUPER]) + int(total[t0] - total[(t0 // SUPER) * SUPER])
        assert first == int(total[t0])
    if len(units) == -(-n_tiles // u):
        assert seen == int(cnt.sum())
