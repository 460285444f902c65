"""The appends kernel's units of massive tiles (csrc/sfp_step.cuh,
sfp_append_units) by the condition that stands in the kernel, at every tile
length that a step can have: powers of two in the steps of three launches,
any multiple of 32 in the one-launch kernel, and those that a map too long for
the counters takes next.  Units hold whole tiles of one super-tile, fit the
warp's list of SFP_TILE_MAX particles, and cover every tile once."""
import os
import re

import numpy as np
import pytest

import sfparticles_b200

CSRC = os.path.join(os.path.dirname(sfparticles_b200.__file__), "csrc")
STEP = open(os.path.join(CSRC, "sfp_step.cuh")).read()
SUPER = int(re.search(r"#define SFP_SUPER_TILE (\d+)", STEP).group(1))
TILE_MAX = int(re.search(r"#define SFP_TILE_MAX (\d+)", open(os.path.join(CSRC, "sfp_run.cuh")).read()).group(1))
RULE = re.search(r"while \((.*)\) U <<= 1;", STEP).group(1)
RULE = (RULE.replace("&&", "and").replace("/", "//").replace("V.mtile", "tile").replace("SFP_TILE_MAX", str(TILE_MAX))
        .replace("SFP_SUPER_TILE", str(SUPER)))


def unit_tiles(n_tiles, n_warps, tile):
    U = 1
    while eval(RULE, {}, dict(nm=n_tiles, nw=n_warps, tile=tile, U=U)):
        U <<= 1
    return U


def next_tiles(tile):
    out = [tile]
    while out[-1] < TILE_MAX:
        out.append(min(2 * out[-1], TILE_MAX))
    return out


@pytest.mark.parametrize("n_warps", [8, 2360, 2368, 3552])
@pytest.mark.parametrize("tile", sorted({t for k in range(32, TILE_MAX + 1, 32) for t in next_tiles(k)}))
def test_units_at_any_tile_length(tile, n_warps):
    assert tile % 32 == 0 and tile <= TILE_MAX
    for n in (1, tile, tile + 1, 40_000, 1_048_577):
        sizes = [n // 3, 0, n - n // 3]  # segments, one empty
        start, acc = [], 0
        for s in sizes:
            acc = -(-acc // SUPER) * SUPER
            start.append(acc)
            acc += -(-s // tile)
        u = unit_tiles(acc, n_warps, tile)
        assert SUPER % u == 0 and tile * u <= TILE_MAX
        t0 = np.arange(-(-acc // u)) * u
        t1 = np.minimum(t0 + u, acc)
        assert np.all(t0 // SUPER == (t1 - 1) // SUPER)
        # particles that the units of a segment hold, by sfp_append_tile's arithmetic
        pos = len(start) - 1 - np.argmax(np.array(start)[::-1, None] <= t0, axis=0)
        base = (t0 - np.array(start)[pos]) * tile
        length = np.minimum(np.array(sizes)[pos] - base, tile * u)
        assert base.max() % 32 == 0 and length.max() <= TILE_MAX
        assert sum(int(x) for x in length if x > 0) == n
