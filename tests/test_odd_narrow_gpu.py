"""Odd rows of up to 31 cells, one lane per cell in FP32, and the widths around:
against the oracle bit for bit."""
import numpy as np
import pytest

from cases import OracleAdapter
from test_lbm_gpu import GpuAdapter
from test_odd_lattices_gpu import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [19, 15])
@pytest.mark.parametrize("shape", [(1, 5, 7), (3, 10, 9), (5, 3, 3), (9, 17, 12), (17, 16, 15), (29, 15, 14),
                                   (31, 18, 13), (33, 12, 11)], ids=str)
def test_fp32_bit_exact(gpu, oracle_built, shape, q):
    case = _case(shape, q, 0.58)
    sim, ora = GpuAdapter(case), OracleAdapter(case)
    for n in (1, 20):
        sim.step(n)
        ora.step(n)
        g, r = sim.readback_field(), ora.readback_field()
        assert np.array_equal(g.view(np.uint32), r.view(np.uint32))
