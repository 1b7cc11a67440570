"""A batch member initialized anew between two batch steps, with as many cells
as before (its arrays may come back at the same addresses) but another shape
and body: the batch must step the new lattice, bit-identical to single
steps, in every launch form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _init(s, shape, body, flow):
    from flowcraft_b200.lbm import LatticeModel, Params, Storage, VoxelGrid
    nx, ny, nz = shape
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[body] = 1
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q19, Storage.FP32)
    s.Reset(Params(tau=0.57, inletVelocity=flow, smagorinskyCs=0.1), True)


@pytest.mark.parametrize("shape", [(8, 1), (4, 2), (8, 0), (0, 1)], ids=str)
def test_member_initialized_anew(gpu, shape):
    from flowcraft_b200.batch import LbmBatch
    from flowcraft_b200.lbm import LbmSolver
    a, b = [LbmSolver(), LbmSolver()], [LbmSolver(), LbmSolver()]
    for side in (a, b):
        _init(side[0], (96, 40, 32), np.s_[10:20, 12:20, 30:40], 0.05)
        _init(side[1], (64, 32, 24), np.s_[8:14, 10:16, 20:26], 0.05)
    batch = LbmBatch(a)
    batch.Config(*shape)
    batch.Step(4)
    for s in b:
        s.Step(None, 4)
    for side in (a, b):  # ny and nz swapped; the body wider, with another boundary list
        _init(side[0], (96, 32, 40), np.s_[4:30, 6:9, 40:70], 0.05)
    batch.Step(6)
    batch.Step(3)
    for x, y in zip(a, b):
        y.Step(None, 9)
        assert np.array_equal(x.SavePopulations().view(np.uint32), y.SavePopulations().view(np.uint32))
    batch.close()
