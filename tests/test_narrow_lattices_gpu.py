"""One and two cells along x: every cell lies on the inlet or outlet plane, and
at nx 2 one pair of the step kernels holds both. Against the oracle, and
batches against single steps."""
import numpy as np
import pytest

from cases import OracleAdapter
from test_lbm_gpu import GpuAdapter, _shape_case

pytestmark = pytest.mark.gpu


def _case(shape, q, reverse):
    params = dict(tau=0.6, inlet_velocity=0.05, smagorinsky_cs=0.12, free_slip_y=True, free_slip_z=False,
                  reverse_flow=reverse)
    return _shape_case(shape, (0.0, 0.0, 0.0, 0.0), params, q)


@pytest.mark.parametrize("reverse", [False, True], ids=["forward", "reverse"])
@pytest.mark.parametrize("q", [19, 15])
@pytest.mark.parametrize("shape", [(1, 9, 8), (2, 9, 8), (2, 17, 3)], ids=str)
def test_fp32_bit_exact(gpu, oracle_built, shape, q, reverse):
    case = _case(shape, q, reverse)
    sim, ora = GpuAdapter(case), OracleAdapter(case)
    for n in (1, 1, 8):
        sim.step(n)
        ora.step(n)
        g, r = sim.readback_field(), ora.readback_field()
        assert np.array_equal(g.view(np.uint32), r.view(np.uint32))


@pytest.mark.parametrize("config", [(4, 1), (8, 2), (16, 1), (8, 0), (0, 1)], ids=str)
@pytest.mark.parametrize("storage", ["FP32", "FP16_OFFSET"])
def test_batch_equals_single_steps(gpu, storage, config):
    from flowcraft_b200.batch import LbmBatch
    from flowcraft_b200.lbm import Storage
    shapes = [(2, 9, 8), (4, 10, 6), (2, 20, 5)]
    a, b = ([GpuAdapter(_case(s, 19, k == 1), storage=Storage[storage]).s for k, s in enumerate(shapes)]
            for _ in range(2))
    batch = LbmBatch(a)
    batch.Config(*config)
    batch.Step(5)
    for x, y in zip(a, b):
        y.Step(None, 5)
        assert np.array_equal(x.SavePopulations().view(np.uint32), y.SavePopulations().view(np.uint32))
    batch.close()
