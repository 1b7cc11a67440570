"""Lattices with odd nx through the pair kernel: pairs shifted on the rows
whose first cell has an odd index, plane stride padded when nx, ny and nz are
all odd. FP32 against the oracle bit for bit; the 16-bit formats against the
FP64 oracle with the tolerances of the even-nx test."""
import numpy as np
import pytest

from cases import OracleAdapter, geometry
from test_lbm_gpu import GpuAdapter, _shape_case

# (nx, ny, nz): every parity of ny and nz, one and several 64-cell chunks, a
# row that ends on, before and after a chunk's end with and without the shift
SHAPES = [(3, 9, 8), (33, 15, 13), (61, 16, 17), (63, 18, 14), (65, 17, 15), (127, 12, 13), (129, 13, 12), (191, 13, 11)]
CELLS = {19: [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1),
              (0, 1, -1)], 15: [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1), (1, 1, -1), (1, -1, 1),
                               (-1, 1, 1)]}


def _case(shape, q, tau):
    nx, ny, nz = shape
    r = 0.2 * min(ny, nz) if nx > 3 else 0.0
    params = dict(tau=tau, inlet_velocity=0.05, smagorinsky_cs=0.12, free_slip_y=nx % 4 == 1, free_slip_z=ny % 2,
                  reverse_flow=nx % 4 == 3)
    return _shape_case(shape, (0.4 * nx, 0.47 * ny, 0.52 * nz, r), params, q)


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_pair_reads_stay_inside_the_set(shape):
    """The addresses pairs_tile forms off the faces, also for the cell of a
    pair that lies outside its row, against the allocation."""
    nx, ny, nz = shape
    n = nx * ny * nz
    ps, guard = n + (n & 1), 64  # 256 guard bytes hold at least 64 elements
    for q, half in CELLS.items():
        dirs = [half[0]] + [tuple(s * v for v in e) for e in half[1:] for s in (1, -1)]
        assert len(dirs) == q
        for row in {(z * ny + y) for z in (1, nz - 2) for y in (1, ny - 2)}:
            sh = row & 1
            for x in (-sh, nx - 2, nx - 1, nx):  # first and last pairs that hold a cell of the row
                if (x + sh) % 2 or x >= nx:
                    continue
                for i, e in enumerate(dirs):
                    a = i * ps + row * nx + x - (e[0] + e[1] * nx + e[2] * nx * ny)
                    assert 0 <= a and a + 1 < q * ps + guard


@pytest.mark.gpu
@pytest.mark.parametrize("q", [19, 15])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_fp32_bit_exact_odd_nx(gpu, oracle_built, shape, q):
    case = _case(shape, q, 0.6)
    sim, ora = GpuAdapter(case), OracleAdapter(case)
    sim.step(21)
    ora.step(21)
    g, r = sim.readback_field(), ora.readback_field()
    assert np.array_equal(g.view(np.uint32), r.view(np.uint32))
    # planes through the layer copy's pitch against the population readout
    import torch
    nx, ny, nz = shape
    pops = sim.s.SavePopulations().reshape(q, nz, ny, nx)
    buf = torch.empty((q, ny, nx), dtype=torch.float32, device="cuda")
    sim.s.LayerCopy(nz // 2, buf.data_ptr(), True)
    sim.s.Sync()
    fluid = ~geometry(case["geom"])[0].astype(bool)[nz // 2]
    assert np.array_equal(buf.cpu().numpy()[:, fluid], pops[:, nz // 2][:, fluid])


@pytest.mark.gpu
@pytest.mark.parametrize("storage,tol", [("FP16_OFFSET", 2e-4), ("BF16_OFFSET", 2e-3)])
@pytest.mark.parametrize("shape", SHAPES[1:], ids=str)
def test_offset_storage_odd_nx_vs_fp64(gpu, oracle_built, shape, storage, tol):
    from flowcraft_b200.lbm import Storage
    case = _case(shape, 19, 0.6)
    sim, ref = GpuAdapter(case, storage=Storage[storage]), OracleAdapter(case, "f64")
    sim.step(30)
    ref.step(30)
    g = sim.readback_field().reshape(-1, 4).astype(np.float64)
    r = ref.o.readback_field_f64().reshape(-1, 4)
    d = np.abs(g - r)[~geometry(case["geom"])[0].ravel().astype(bool)]
    assert np.isfinite(g).all() and d[:, 0].max() < tol and d[:, 1:].max() < tol
