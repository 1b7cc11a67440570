"""The odd-nx 16-bit kernels' packed two-cell collision against the one-cell
one, through the step: a cell next to a wall cell's neighbour is updated alone,
the same cell without the wall as half of a pair, from the same populations.
Bit for bit; and D3Q15 against the FP64 oracle with the D3Q19 test's
tolerances."""
import numpy as np
import pytest

from cases import OracleAdapter, geometry
from test_lbm_gpu import GpuAdapter
from test_odd_lattices_gpu import SHAPES, _case

pytestmark = pytest.mark.gpu


def _step(shape, q, storage, solid, pops):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, VoxelGrid
    nx, ny, nz = shape
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, solid=solid), LatticeModel.D3Q15 if q == 15 else LatticeModel.D3Q19,
                  Storage[storage])
    s.Reset(Params(tau=0.53, inletVelocity=0.05, smagorinskyCs=0.17), True)
    s.LoadPopulations(pops)
    s.Step(None, 1)
    return s.SavePopulations().reshape(q, nz, ny, nx)


@pytest.mark.parametrize("storage", ["FP16_OFFSET", "BF16_OFFSET"])
@pytest.mark.parametrize("shape", [(257, 31, 29), (257, 30, 29)], ids=str)
@pytest.mark.parametrize("q", [19, 15])
def test_pair_collision_equals_single_cells(gpu, shape, q, storage):
    nx, ny, nz = shape
    rng = np.random.default_rng(q + ny)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12 if q == 19 else [2 / 9] + [1 / 9] * 6 + [1 / 72] * 8)
    pops = (w[:, None] * (1.0 + rng.uniform(-0.12, 0.12, (q, nx * ny * nz)))).astype(np.float32).ravel()
    wall = np.zeros((nz, ny, nx), np.uint8)
    wall[3:-3:4, 3:-3:4, 65:190:5] = 1
    far = np.ones((nz, ny, nx), bool)  # no wall cell in the 3x3x3 around
    for z, y, x in np.argwhere(wall):
        far[z - 1:z + 2, y - 1:y + 2, x - 1:x + 2] = False
    alone = far & ~(np.roll(far, 1, 2) & np.roll(far, -1, 2))  # beside a cell of the boundary list
    assert alone.sum() > 2000
    a = _step(shape, q, storage, np.zeros_like(wall), pops)
    b = _step(shape, q, storage, wall, pops)
    assert np.array_equal(a[:, alone].view(np.uint32), b[:, alone].view(np.uint32))
    assert np.array_equal(a[:, far].view(np.uint32), b[:, far].view(np.uint32))


@pytest.mark.parametrize("storage,tol", [("FP16_OFFSET", 2e-4), ("BF16_OFFSET", 2e-3)])
@pytest.mark.parametrize("shape", SHAPES[1:], ids=str)
def test_offset_storage_d3q15_vs_fp64(gpu, oracle_built, shape, storage, tol):
    from flowcraft_b200.lbm import Storage
    case = _case(shape, 15, 0.6)
    sim, ref = GpuAdapter(case, storage=Storage[storage]), OracleAdapter(case, "f64")
    sim.step(30)
    ref.step(30)
    g = sim.readback_field().reshape(-1, 4).astype(np.float64)
    r = ref.o.readback_field_f64().reshape(-1, 4)
    d = np.abs(g - r)[~geometry(case["geom"])[0].ravel().astype(bool)]
    assert np.isfinite(g).all() and d[:, 0].max() < tol and d[:, 1:].max() < tol
