"""The voxelizer's tiled raster and flood fill at the sizes where tiles are
cut: grids whose sides are not multiples of the 8-cell tile, the 4-cell warp
box or the finalize pass's four cells, triangle soups that leave many pockets
and corridors (runs that meet only across rows, layers or tile faces), and
grids whose cell 0 is inside the surface. Bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 40), (7, 1, 1), (8, 8, 8), (9, 17, 8), (33, 31, 7), (64, 10, 23), (130, 5, 19), (41, 40, 39)]


def _soup(dims, count, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    # world x spans grid y, world y spans grid x
    size = np.array([ny, nx, nz], np.float64)
    centre = rng.uniform(-0.1, 1.1, (count, 1, 3)) * size
    pos = centre + rng.uniform(-1, 1, (count, 3, 3)) * np.maximum(0.35 * size, 1.5)
    return pos.reshape(-1, 3).astype(np.float32), np.arange(3 * count, dtype=np.uint32)


@pytest.mark.parametrize("count", [0, 1, 12, 60])
@pytest.mark.parametrize("dims", DIMS, ids=str)
def test_soup_matches_oracle(gpu, oracle_built, dims, count):
    from flowcraft_b200.voxelizer import VoxelizeOnGrid
    for seed in range(3):
        pos, idx = _soup(dims, max(count, 1), 100 * count + seed)
        idx = idx if count else idx[:0]
        want_s, want_d = oracle_built.voxelize(pos, idx, dims, 1.0, np.zeros(3, np.float32))
        g = VoxelizeOnGrid(pos, idx, dims, 1.0, (0.0, 0.0, 0.0), device=0)
        assert np.array_equal(g.solid.cpu().numpy(), want_s.ravel())
        assert np.array_equal(g.signedDistance.cpu().numpy().view(np.uint32), want_d.ravel().view(np.uint32))
