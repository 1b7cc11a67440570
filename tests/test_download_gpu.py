"""Blocking downloads in chunks around the staging ring: one chunk, a cell
more or less than one, a full ring, more chunks than slots, a range of layers,
and the trails, against the one-copy asynchronous readback and a per-layer
readback."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 16 bytes per cell: chunks are 1 MiB up to 8 MiB, eight slots
SHAPES = [(64, 32, 32), (65, 33, 31), (63, 32, 32), (128, 128, 33), (256, 128, 128), (261, 131, 127)]


def _solver(shape):
    from flowcraft_b200.lbm import LbmSolver, Params, Storage, VoxelGrid
    nx, ny, nz = shape
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[nz // 3:nz // 2, ny // 3:ny // 2, nx // 3:nx // 3 + 3] = 1
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), storage=Storage.FP16_OFFSET)
    s.Reset(Params(tau=0.6, inletVelocity=0.05, smagorinskyCs=0.1), True)
    s.Step(None, 4)
    return s


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_blocking_readback_equals_async(gpu, shape):
    s = _solver(shape)
    nx, ny, nz = shape
    want = np.empty(4 * nx * ny * nz, np.float32)
    s.ReadbackFieldAsync(want)
    s.ReadbackWait()
    for _ in range(2):
        assert np.array_equal(s.ReadbackField().view(np.uint32), want.view(np.uint32))
    part = np.zeros_like(want)
    s.ReadbackFieldRange(1, nz - 2, part)
    layer = 4 * nx * ny
    assert np.array_equal(part[layer:-layer].view(np.uint32), want[layer:-layer].view(np.uint32))
    assert not part[:layer].any() and not part[-layer:].any()


@pytest.mark.parametrize("count,length", [(3, 5), (20000, 48), (1 << 17, 61)])
def test_trails_of_any_size(gpu, count, length):
    from flowcraft_b200.smoke import SmokeTrailSystem
    s = _solver((64, 32, 32))
    smoke = SmokeTrailSystem(s)
    smoke.Reset(False, count, length)
    pos = np.random.default_rng(1).uniform(2, 20, (count, 3)).astype(np.float32)
    smoke.SetPositions(pos)
    points, lens = smoke.Trails()
    assert np.array_equal(points[:, 0], pos) and not points[:, 1:].any() and (lens == 1).all()
