"""A blocking readback behind a second of queued steps waits without keeping a
core busy, also when it takes more chunks than the staging buffer has slots."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_readback_behind_queued_steps_sleeps(gpu):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, VoxelGrid
    nx, ny, nz = 512, 256, 256
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=np.zeros((nz, ny, nx), np.uint8)), LatticeModel.D3Q19,
                  Storage.FP16_OFFSET)
    s.Reset(Params(tau=0.6, inletVelocity=0.05, smagorinskyCs=0.1), True)
    s.ReadbackField()
    wall, cpu = [], []
    for steps in (0, 2000):  # 2000 steps are about 1.1 s on the device
        s.Step(None, steps)
        t, c = time.perf_counter(), time.process_time()
        s.ReadbackField()
        wall.append(time.perf_counter() - t)
        cpu.append(time.process_time() - c)
    queued = wall[1] - wall[0]
    assert queued > 0.3
    assert cpu[1] - cpu[0] < 0.4 * queued, (wall, cpu)
