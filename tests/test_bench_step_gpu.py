"""The bench times the steps a program takes: one launch each on a lattice of
this size, and the time of LbmSolver.Step."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.abspath(os.path.join(os.path.dirname(__file__), "..")))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["fp16_offset", "fp16_learned", "fp32_aa"])
def test_bench_times_the_shipped_step(gpu, variant):
    import bench
    args = bench.parse_args(["--steps", "50", "--warmup", "20", "--spinup", "20"])
    cfg = dict(bench.CONFIGS["c1"])
    solid, sdf = bench.build_geometry(cfg, "cuda:0")
    r = bench.time_variant(args, cfg, solid, sdf, variant, 0, False, False)
    assert r["launches"] == 50
    s = bench.make_solver(cfg, solid, sdf, variant, 0)
    s.Step(None, 40)
    s.Sync()
    ms = min(bench.timed_steps(s, 50) for _ in range(3))
    assert np.isclose(r["total_ms"], ms, rtol=0.25), (r["total_ms"], ms)
    s.close()
