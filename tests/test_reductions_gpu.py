"""The statistics and force reductions at the sizes where their 128-cell
groups are cut: fewer cells than a group, a cell more or less than several,
more solid cells than a group or a queue holds, rows that keep a body in the
same part of every group, and a wall that fills a lattice but for one layer.
Against sums over the field the solver reads back (bit-exact to the oracle
elsewhere), FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(5, 3, 4), (8, 4, 4), (16, 8, 1), (43, 3, 1), (129, 1, 1), (64, 16, 16), (512, 9, 8), (127, 33, 31)]


def _solver(shape, body, q, storage, streaming):
    from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, Streaming, VoxelGrid
    nx, ny, nz = shape
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    if body == "block":
        solid = (x >= nx // 3) & (x <= nx // 2) & (y < (ny + 1) // 2)
    elif body == "filled":
        solid = (z > 0) | (y > 0)
    else:
        solid = np.zeros((nz, ny, nx), bool)
    s = LbmSolver()
    assert s.Init(0, VoxelGrid(nx, ny, nz, 2.0, (1.0, -3.0, 0.5), solid.astype(np.uint8), None),
                  LatticeModel.D3Q19 if q == 19 else LatticeModel.D3Q15, Storage[storage], Streaming[streaming])
    s.Reset(Params(tau=0.7, inletVelocity=0.05, smagorinskyCs=0.1), True)
    s.Step(None, 5)
    return s, solid.ravel()


@pytest.mark.parametrize("body", ["none", "block", "filled"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("q,storage,streaming", [(19, "FP32", "PINGPONG"), (15, "FP16_OFFSET", "PINGPONG"),
                                                 (19, "FP16_OFFSET", "AA")])
def test_sums_match_the_field(gpu, shape, body, q, storage, streaming):
    nx, ny, nz = shape
    if streaming == "AA" and (nx % 2 or nx < 4):
        pytest.skip("in-place streaming needs an even nx of at least 4")
    s, solid = _solver(shape, body, q, storage, streaming)
    f = s.ReadbackField().reshape(-1, 4).astype(np.float64)
    st, a = s.ReadbackStats(), s.AerodynamicForces()
    fl, so = f[~solid], f[solid]
    sp = np.sqrt((s.ReadbackField().reshape(-1, 4)[~solid][:, 1:] ** 2).sum(1, dtype=np.float32)).astype(np.float64)
    assert st.fluidCells == len(fl) and a.solidCells == len(so)
    # FP64 sums of float values: only the order differs (speeds are rounded
    # once more, in float, by either side)
    assert abs(st.totalMass - fl[:, 0].sum()) <= 1e-12 * len(fl)
    assert abs(st.extra["speed_sum"] - sp.sum()) <= 3e-7 * max(sp.sum(), 1e-30)
    if len(fl):
        assert st.minDensity == np.float32(fl[:, 0].min()) and st.maxDensity == np.float32(fl[:, 0].max())
    for got in (st.forceSum, a.forceSum):
        assert np.abs(np.array(got) - so[:, 1:].sum(0)).max(initial=0.0) <= 1e-12 * max(np.abs(so).sum(), 1e-30)
    if len(so):
        idx = np.nonzero(solid)[0]
        at = np.stack([(idx // nx) % ny, idx % nx, idx // (nx * ny)], 1) + 0.5
        pos = np.array([1.0, -3.0, 0.5]) + 2.0 * at
        lift = np.abs(so[:, 3])
        if lift.sum() > 1e-9:
            want = (lift[:, None] * pos).sum(0) / lift.sum()
            assert np.abs(np.array(a.centerOfPressure) - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
            g = np.clip(np.floor((want[[1, 0]] - np.array([-3.0, 1.0])) / 2.0).astype(int), 0, [nx - 1, ny - 1])
            near = np.abs((want[[1, 0]] - np.array([-3.0, 1.0])) / 2.0 - np.round((want[[1, 0]] - [-3.0, 1.0]) / 2.0))
            if near.min() > 1e-4:  # the patch's centre cell does not hang on rounding
                cols = solid.reshape(nz, ny, nx)[:, np.clip(np.arange(g[1] - 2, g[1] + 3), 0, ny - 1)][
                    :, :, np.clip(np.arange(g[0] - 2, g[0] + 3), 0, nx - 1)]
                top = np.nonzero(cols.any(axis=(1, 2)))[0]
                eff = top.max() if len(top) else idx.max() // (nx * ny)
                assert abs(a.liftArrowBase[2] - (0.5 + 2.0 * (eff + 1))) < 1e-5
