"""Lattices as tall as a launch holds (65,535 layers): the boundary list's
blocks do not fit into the launch beside the layers, or not into one launch
at all, and go out on their own. Against steps over shorter layer ranges,
whose blocks all fit (in place: whose list fits), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the last shape's list alone is longer than one launch's blocks
CASES = [((4, 3, 65535), "FP32", "PINGPONG", False), ((4, 3, 65535), "FP16_OFFSET", "AA", False),
         ((5, 3, 65535), "BF16_OFFSET", "PINGPONG", False), ((6, 4, 65534), "FP16_OFFSET", "PINGPONG", True),
         ((4, 3, 65535), "FP16_OFFSET", "AA", True), ((64, 8, 65535), "FP16_OFFSET", "PINGPONG", False)]


def _solver(shape, storage, streaming, learned):
    from flowcraft_b200.closure import ClosureWeights
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, Streaming, VoxelGrid
    nx, ny, nz = shape
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[1::4, 1::2, 1::2] = 1
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q19, Storage[storage], Streaming[streaming])
    s.Reset(Params(tau=0.6, inletVelocity=0.05, smagorinskyCs=0.1), True)
    if learned:
        s.SetClosure(ClosureWeights.random(3))
    return s, solid


@pytest.mark.parametrize("shape,storage,streaming,learned", CASES)
def test_step_of_a_tall_lattice(gpu, shape, storage, streaming, learned):
    a, solid = _solver(shape, storage, streaming, learned)
    b, _ = _solver(shape, storage, streaming, learned)
    entries = a.BoundaryInfo()["boundary_cells"]
    blocks = ((shape[0] + 63) // 64) * ((shape[1] + 7) // 8)
    assert shape[2] + -(-entries // (256 * blocks)) > 65535
    assert shape[0] < 64 or entries > 65535 * 256
    for _ in range(3):
        a.Step(None, 1)
        for z in range(0, shape[2], 20000):
            b.StepRange(None, z, min(20000, shape[2] - z))
        b.AdvanceSubstep()
    assert np.array_equal(a.ReadbackField().view(np.uint32), b.ReadbackField().view(np.uint32))
    assert a.ReadbackStats().valid and not a.HasDiverged()
