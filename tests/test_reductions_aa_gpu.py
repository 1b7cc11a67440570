"""Statistics and forces of in-place states, after odd and even steps, against
ping-pong's on the same flow: cells on every face, edge and corner, rows that
end inside a group of 128 cells. Extremes, counts and cells are equal; the FP64
sums run in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(4, 3, 3), (4, 1, 9), (34, 7, 5), (66, 33, 17), (130, 20, 9), (256, 3, 40)]


def _solver(shape, q, storage, streaming):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, Streaming, VoxelGrid
    nx, ny, nz = shape
    solid = np.zeros((nz, ny, nx), np.uint8)
    if ny > 4:
        solid[nz // 3:nz // 2, ny // 3:ny // 2, nx // 3:nx // 3 + 3] = 1
        solid[0, 0, nx // 2:nx // 2 + 2] = 1
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q15 if q == 15 else LatticeModel.D3Q19,
                  Storage[storage], Streaming[streaming])
    s.Reset(Params(tau=0.56, inletVelocity=0.06, smagorinskyCs=0.1), True)
    return s


@pytest.mark.parametrize("storage", ["FP32", "FP16_OFFSET"])
@pytest.mark.parametrize("q", [19, 15])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_in_place_reductions_equal_ping_pong(gpu, shape, q, storage):
    a, b = _solver(shape, q, storage, "AA"), _solver(shape, q, storage, "PINGPONG")
    for _ in range(4):
        a.Step(None, 1)
        b.Step(None, 1)
        x, y = a.ReadbackStats(), b.ReadbackStats()
        for k in ("minDensity", "maxDensity", "maxSpeed", "maxStress", "fluidCells", "hasNaN"):
            assert getattr(x, k) == getattr(y, k), k
        for k in ("totalMass", "avgDensity", "avgSpeed", "forceX"):
            assert np.isclose(getattr(x, k), getattr(y, k), rtol=1e-6, atol=1e-9), k
        f, g = a.AerodynamicForces(), b.AerodynamicForces()
        assert (f.minStress, f.maxStress) == (g.minStress, g.maxStress)
        assert np.isclose(f.forceX, g.forceX, rtol=1e-6, atol=1e-9)
