"""Batches stepped by the members' own kernels (rows 0): more members than
streams, so that a chain runs through several lattices; members large enough
for direct launches; calls long enough for the graph of many steps, with a
remainder; a pending asynchronous readback. Bit-identical to single steps."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _make(shapes, storage="FP16_OFFSET"):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, VoxelGrid
    out = []
    for k, (nx, ny, nz) in enumerate(shapes):
        solid = np.zeros((nz, ny, nx), np.uint8)
        solid[nz // 3:nz // 2, ny // 3:ny // 2, nx // 4 + k % 3:nx // 3 + 1 + k % 3] = 1
        s = LbmSolver()
        assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q19, Storage[storage])
        s.Reset(Params(tau=0.56 + 0.002 * k, inletVelocity=0.05, smagorinskyCs=0.1, reverseFlow=k % 4 == 3), True)
        out.append(s)
    return out


SMALL = [(16 + 2 * (k % 7), 9 + k % 5, 8 + k % 3) for k in range(40)]
LARGE = [(128, 32, 32 + k % 2) for k in range(20)]  # from 2^17 cells
# calls of 20 members: direct up to 51 steps, above that graphs of 12 steps and the rest
SETS = {"small": (SMALL, (1, 2, 7, 30)), "small_odd_then_even": (SMALL, (3, 4)), "large_direct": (LARGE[:4], (5, 2, 7)),
        "large_chains": (LARGE, (3, 4)), "large_graph": (LARGE, (60, 61)), "few_graph": (SMALL[:3], (520,))}


@pytest.mark.parametrize("name", SETS)
def test_members_equal_single_steps(gpu, name):
    from flowcraft_b200.batch import LbmBatch
    shapes, calls = SETS[name]
    a, b = _make(shapes), _make(shapes)
    batch = LbmBatch(a)
    batch.Config(0, 1)
    for n in calls:
        batch.Step(n)
    for x, y in zip(a, b):
        y.Step(None, sum(calls))
        assert np.array_equal(x.SavePopulations().view(np.uint32), y.SavePopulations().view(np.uint32))
    batch.close()


@pytest.mark.parametrize("shapes,n", [(SMALL[:20], 9), (LARGE, 3), (LARGE, 60)], ids=["small", "large", "graph"])
def test_member_with_pending_readback(gpu, shapes, n):
    from flowcraft_b200.batch import LbmBatch
    a, b = _make(shapes), _make(shapes)
    batch = LbmBatch(a)
    batch.Config(0, 1)
    batch.Step(4)
    for s in b:
        s.Step(None, 4)
    out = np.empty(4 * a[1].CellCount(), np.float32)
    a[1].ReadbackFieldAsync(out)
    batch.Step(n)
    a[1].ReadbackWait()
    assert np.array_equal(out.view(np.uint32), b[1].ReadbackField().ravel().view(np.uint32))
    for x, y in zip(a, b):
        y.Step(None, n)
        assert np.array_equal(x.SavePopulations().view(np.uint32), y.SavePopulations().view(np.uint32))
    batch.close()


def test_long_call_returns_early(gpu):
    """24,000 launches one by one would hold the caller for most of the call."""
    from flowcraft_b200.batch import LbmBatch
    a = _make([(128, 64, 32)] * 16)
    batch = LbmBatch(a)
    batch.Config(0, 1)
    batch.Step(1500)
    for s in a:
        s.Sync()
    t = time.perf_counter()
    batch.Step(1500)
    host = time.perf_counter() - t
    for s in a:
        s.Sync()
    assert host < 0.25 * (time.perf_counter() - t)
    batch.close()
