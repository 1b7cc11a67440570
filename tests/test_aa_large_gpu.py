"""In-place FP32 lattices on both sides of the size from which the boundary
list runs in a launch of its own, against ping-pong, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(shape, q, streaming):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, Streaming, VoxelGrid
    nx, ny, nz = shape
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[nz // 3:nz // 2, ny // 3:ny // 2, nx // 3:nx // 3 + 9] = 1
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q15 if q == 15 else LatticeModel.D3Q19,
                  Storage.FP32, Streaming[streaming])
    s.Reset(Params(tau=0.56, inletVelocity=0.06, smagorinskyCs=0.1), True)
    return s


@pytest.mark.parametrize("shape,q,per_step", [((256, 182, 180), 15, 1), ((256, 182, 181), 15, 2),
                                              ((512, 256, 255), 19, 1), ((512, 256, 256), 19, 2)], ids=str)
def test_in_place_equals_ping_pong(gpu, shape, q, per_step):
    a, b = _solver(shape, q, "AA"), _solver(shape, q, "PINGPONG")
    for n in (5, 4):
        before = a.LaunchCount()
        a.Step(None, n)
        assert a.LaunchCount() - before == n * per_step
        b.Step(None, n)
    assert np.array_equal(a.ReadbackField().view(np.uint32), b.ReadbackField().view(np.uint32))
