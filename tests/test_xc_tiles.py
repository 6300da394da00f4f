"""The XC flow's cut of a grid into tiles."""
import pytest

from pyscf_wb97mv_fast_gb300.gpu.xc import OVERLAP_TILE_PTS, _tiles


@pytest.mark.parametrize('n', [0, 1, 32, OVERLAP_TILE_PTS, 2 * OVERLAP_TILE_PTS - 1,
                               2 * OVERLAP_TILE_PTS, 3 * OVERLAP_TILE_PTS + 7,
                               4 * OVERLAP_TILE_PTS + 2047, 40 * OVERLAP_TILE_PTS + 1])
@pytest.mark.parametrize('tile_pts', [1, 4096, 50000, 1 << 40])
def test_tiles_cover_the_grid(n, tile_pts):
    tiles = _tiles(n, tile_pts)
    assert [i for t in tiles for i in t] == sorted(i for t in tiles for i in t)
    assert sum(b - a for a, b in tiles) == n and all(b > a for a, b in tiles)
    assert all(tiles[i][1] == tiles[i + 1][0] for i in range(len(tiles) - 1))
    assert all(b - a <= max(32, tile_pts) for a, b in tiles)
    if tile_pts > n:
        assert len(tiles) <= (1 if n < 2 * OVERLAP_TILE_PTS else 4)
        assert all((b - a) % 2048 == 0 for a, b in tiles[:-1])
