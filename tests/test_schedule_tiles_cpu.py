"""The pair kernel's schedules as they are launched, host arithmetic only: on a single grid the rule for grids of at
least four items per CTA, and below that the rule for small ones (chunks of 1 to nz planes by the stated cost);
and the items of a stack in 32 x 16 tiles as in 64-column ones. Every plane of every tile belongs to one item."""
import math

import numpy as np
import pytest

from em_lab_gb300 import grid

TILES = [(64, 4), (64, 8), (64, 16), (32, 16)]
CTAS = [3 * 152, 2 * 152, 152, 7]
SHAPES = [(48, 40, 9), (70, 37, 3), (64, 8, 1), (48, 48, 48), (96, 96, 96), (128, 128, 128), (211, 147, 93), (24, 24, 3000),
          (192, 192, 128), (320, 300, 280), (384, 384, 256), (512, 512, 512), (1000, 20, 1000), (1, 1, 1), (1, 1, 5000)]


@pytest.mark.parametrize("cols,rows", TILES)
@pytest.mark.parametrize("shape", SHAPES)
def test_launched_schedule(shape, cols, rows):
    nx, ny, nz = shape
    tiles = -(-nx // cols) * -(-ny // rows)
    for ctas in CTAS:
        zc, items = grid.pair_launch(nx, ny, nz, cols, rows, ctas)
        chunks = -(-nz // zc)
        # whole chunks of zc planes, the last one not empty: every plane of every tile once
        assert 1 <= zc <= nz and (chunks - 1) * zc < nz and items == chunks * tiles
        if cols == 64:
            large = grid.pair_schedule(nx, ny, nz, rows, ctas)
            if large[1] >= 4 * ctas:
                assert (zc, items) == large
                continue
        # the small grids' rule: the first chunk length of the least cost
        def cost(z):
            n = -(-nz // z) * tiles
            return (z + 2.5) * (0.5 * (n / ctas) + 0.5 * -(-n // ctas) + 0.75)
        if items < 4 * ctas or cols == 64:
            best = min(cost(z) for z in range(1, nz + 1))
            assert math.isclose(cost(zc), best, rel_tol=1e-12)


@pytest.mark.parametrize("seed", range(4))
def test_narrow_ragged_items_cover_every_cell_once(seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 24))
    nx, ny, nz = rng.integers(1, 200, n), rng.integers(1, 200, n), rng.integers(1, 160, n)
    z0 = np.concatenate([[0], np.cumsum(nz + 1)[:-1]])
    for ctas in CTAS:
        x0, y0, zs, ze, sc = grid.ragged_items(z0, nx, ny, nz, 16, ctas, tile_cols=32).T
        assert (np.diff(sc) >= 0).all()
        for s in range(n):
            m = sc == s
            covered = np.zeros((nz[s], -(-ny[s] // 16), -(-nx[s] // 32)), int)
            assert (x0[m] % 32 == 0).all() and (y0[m] % 16 == 0).all() and (x0[m] < nx[s]).all() and (y0[m] < ny[s]).all()
            for x, y, a, b in zip(x0[m], y0[m], zs[m] - z0[s], ze[m] - z0[s]):
                assert 0 <= a < b <= nz[s]
                covered[a:b, y // 16, x // 32] += 1
            assert (covered == 1).all()


def test_other_tiles_are_refused():
    for cols, rows in ((32, 8), (64, 6), (48, 16), (0, 16)):
        with pytest.raises(grid.EmlabError):
            grid.pair_launch(64, 64, 64, cols, rows, 304)
        with pytest.raises(grid.EmlabError):
            grid.ragged_items([0], [8], [8], [8], rows, 304, tile_cols=cols)
    with pytest.raises(grid.EmlabError):
        grid.pair_launch(64, 64, 0, 64, 8, 304)
