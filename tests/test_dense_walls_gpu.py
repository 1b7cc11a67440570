"""Lattices with more than 2^20 boundary-list entries, which run in a launch of
their own, against steps over layer ranges, whose lists run in the step
kernel: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(shape, q, storage):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, VoxelGrid
    nx, ny, nz = shape
    solid = (np.random.default_rng(7).random((nz, ny, nx)) < 0.2).astype(np.uint8)
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q15 if q == 15 else LatticeModel.D3Q19,
                  Storage[storage])
    s.Reset(Params(tau=0.6, inletVelocity=0.03, smagorinskyCs=0.1), True)
    return s


@pytest.mark.parametrize("shape,q,storage", [((160, 96, 96), 19, "FP16_OFFSET"), ((160, 96, 96), 19, "FP32"),
                                             ((161, 97, 95), 19, "BF16_OFFSET"), ((161, 97, 95), 15, "FP32")], ids=str)
def test_list_apart_equals_list_inside(gpu, shape, q, storage):
    a, b = _solver(shape, q, storage), _solver(shape, q, storage)
    assert a.BoundaryInfo()["boundary_cells"] >= 1 << 20
    before = a.LaunchCount()
    a.Step(None, 6)
    assert a.LaunchCount() - before == 12
    for _ in range(6):
        before = b.LaunchCount()
        for z in range(0, shape[2], 40):
            b.StepRange(None, z, min(40, shape[2] - z))
        assert b.LaunchCount() - before == 3
        b.AdvanceSubstep()
    assert np.array_equal(a.SavePopulations().view(np.uint32), b.SavePopulations().view(np.uint32))
