"""Chained steps (a step kernel starting under the end of the one before)
against steps issued one at a time: small lattices where several steps could
overlap, ones whose layers hold no bulk cell, long chains, a pending readback
in the middle, and a chain captured into a graph. Bit-identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMATS = [("FP32", "PINGPONG", False), ("FP16_OFFSET", "PINGPONG", False), ("FP16_OFFSET", "PINGPONG", True),
           ("FP32", "AA", False), ("BF16_OFFSET", "AA", False), ("FP16_OFFSET", "AA", True)]
SHAPES = [(8, 3, 3), (48, 24, 24), (64, 40, 5), (130, 33, 31)]


def _solver(shape, storage, streaming, learned, walls):
    from flowcraft_b200.closure import ClosureWeights
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, Streaming, VoxelGrid
    nx, ny, nz = shape
    solid = np.zeros((nz, ny, nx), np.uint8)
    solid[nz // 3:nz // 2, ny // 3:ny // 2, nx // 3:nx // 3 + 2] = 1
    if walls:  # whole layers without a fluid cell
        solid[:nz // 2] = 1
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q19, Storage[storage], Streaming[streaming])
    s.Reset(Params(tau=0.56, inletVelocity=0.06, smagorinskyCs=0.1), True)
    if learned:
        s.SetClosure(ClosureWeights.random(3))
    return s


@pytest.mark.parametrize("walls", [False, True], ids=["body", "walls"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("storage,streaming,learned", FORMATS)
def test_chain_equals_single_steps(gpu, shape, storage, streaming, learned, walls):
    a, b = (_solver(shape, storage, streaming, learned, walls) for _ in range(2))
    for n in (2, 3, 64):
        a.Step(None, n)
        for _ in range(n):
            b.Step(None, 1)
            b.Sync()
    assert np.array_equal(a.SavePopulations().view(np.uint32), b.SavePopulations().view(np.uint32))


def test_chain_with_pending_readback(gpu):
    a, b = (_solver((128, 64, 48), "FP16_OFFSET", "PINGPONG", False, False) for _ in range(2))
    out = np.empty(4 * a.CellCount(), np.float32)
    a.Step(None, 5)
    a.ReadbackFieldAsync(out)
    a.Step(None, 40)
    b.Step(None, 5)
    want = b.ReadbackField()
    b.Step(None, 40)
    a.ReadbackWait()
    assert np.array_equal(out.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(a.ReadbackField().view(np.uint32), b.ReadbackField().view(np.uint32))


def test_chain_under_capture(gpu):
    cu = pytest.importorskip("cuda.bindings.driver")
    a, b = (_solver((64, 24, 20), "FP32", "PINGPONG", False, False) for _ in range(2))
    b.Sync()
    stream = cu.CUstream(b.Stream())
    assert cu.cuStreamBeginCapture(stream, cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL)[0] == 0
    b.Step(None, 4)
    err, graph = cu.cuStreamEndCapture(stream)
    assert err == 0
    err, ex = cu.cuGraphInstantiate(graph, 0)
    assert err == 0
    for _ in range(3):
        assert cu.cuGraphLaunch(ex, stream)[0] == 0
    a.Step(None, 12)
    assert np.array_equal(a.ReadbackField().view(np.uint32), b.ReadbackField().view(np.uint32))
    cu.cuGraphExecDestroy(ex)
    cu.cuGraphDestroy(graph)
