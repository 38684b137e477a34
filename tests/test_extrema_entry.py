"""The extrema entry's own route (the kernels' knots-only forms) against the CPU oracle: end tiles
of every number of knots around the six that decide the end rule in the tile, rows around the 256
tiles whose tables are in shared memory, dense and empty tiles."""
import numpy as np
import pytest

from test_tile_paths import TILE, _zigzag

pytestmark = pytest.mark.gpu


def _check(pkg, orc, cuda, rows):
    import torch
    got = [t.cpu().numpy() for t in pkg.extrema(torch.tensor(rows, device=cuda))]
    cnt = got[4]
    for r in range(rows.shape[0]):
        for kind in (0, 1):
            ox, oy = orc.extrema(rows[r], kind)
            oy = orc.boundary(ox, oy, kind)
            k = cnt[kind, r]
            assert k == ox.size
            assert np.array_equal(got[2 * kind][r, :k], ox)
            assert np.array_equal(got[2 * kind + 1][r, :k], oy)


@pytest.mark.parametrize("n", [4, 17, TILE, 2 * TILE + 1, 4 * TILE + 700])
def test_extrema_of_every_density(pkg, orc, cuda, n):
    _check(pkg, orc, cuda, np.stack([_zigzag(n, k, 13 * k + n)
                                     for k in (0, 1, 2, 5, 12, 33, 700, 1900, 2048)]))


@pytest.mark.parametrize("few", [0, 1, 2, 4, 6, 8, 10, 11, 12, 13])
def test_extrema_with_sparse_end_tiles(pkg, orc, cuda, few):
    n = 4 * TILE + 700
    rows = []
    for side in range(3):
        row, end = _zigzag(n, 90, few), _zigzag(n, few, 1000 + few)
        if side != 1:
            row[:TILE] = end[:TILE]
        if side != 0:
            row[4 * TILE:] = end[4 * TILE:]
        rows.append(row)
    rows.append(_zigzag(n, 1, few))  # every tile
    _check(pkg, orc, cuda, np.stack(rows))


@pytest.mark.parametrize("n", [256 * TILE, 256 * TILE + 1, 300 * TILE + 77])
def test_extrema_of_long_rows(pkg, orc, cuda, n):
    _check(pkg, orc, cuda, np.stack([_zigzag(n, 40, n), _zigzag(n, 1, n + 1)]))
