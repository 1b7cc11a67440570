"""Grids thinner than a tile along one or two axes: fewer flood-fill nodes per
tile. Bit-identical to the oracle, and scratch memory of a few bytes per cell
where every tile holds a triangle."""
import numpy as np
import pytest

from test_voxelizer_tiles_gpu import _soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 1, 9), (1, 50, 3), (2, 3, 77), (130, 70, 1), (1, 8, 64), (9, 1, 17), (3, 40, 40),
                                  (40, 7, 40), (40, 40, 2)], ids=str)
def test_thin_grids_match_oracle(gpu, oracle_built, dims):
    from flowcraft_b200.voxelizer import VoxelizeOnGrid
    for seed in range(4):
        pos, idx = _soup(dims, 4 + 8 * seed, seed)
        want_s, want_d = oracle_built.voxelize(pos, idx, dims, 1.0, np.zeros(3, np.float32))
        g = VoxelizeOnGrid(pos, idx, dims, 1.0, (0.0, 0.0, 0.0), device=0)
        assert np.array_equal(g.solid.cpu().numpy(), want_s.ravel())
        assert np.array_equal(g.signedDistance.cpu().numpy().view(np.uint32), want_d.ravel().view(np.uint32))


def test_scratch_of_a_plate(gpu):
    cu = pytest.importorskip("cuda.bindings.driver")
    import torch
    from flowcraft_b200.voxelizer import VoxelizeOnGrid
    dims = (2048, 2048, 1)
    pos = torch.tensor([[0, 0, 0.2], [2048, 0, 0.4], [2048, 2048, 0.6], [0, 2048, 0.3]], device="cuda")
    idx = torch.tensor([0, 1, 2, 0, 2, 3], dtype=torch.int32, device="cuda")
    VoxelizeOnGrid(pos, idx, dims, 1.0, (0.0, 0.0, 0.0), device=0)
    torch.cuda.synchronize()
    err, pool = cu.cuDeviceGetDefaultMemPool(0)
    high = cu.CUmemPool_attribute.CU_MEMPOOL_ATTR_USED_MEM_HIGH
    if err or cu.cuMemPoolSetAttribute(pool, high, cu.cuuint64_t(0))[0]:
        pytest.skip("no pool attributes")
    VoxelizeOnGrid(pos, idx, dims, 1.0, (0.0, 0.0, 0.0), device=0)
    torch.cuda.synchronize()
    used = int(cu.cuMemPoolGetAttribute(pool, high)[1])
    assert 0 < used < 10 * 2048 * 2048, used / 2048 ** 2
