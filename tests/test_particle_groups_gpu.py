"""Particle counts around the eight-lane groups and their blocks of sixteen,
with neighbouring groups that advect, leave the grid and sit in the body:
each trail as the numpy restatement advects it, bit for bit, and as the same
particle moves alone."""
import numpy as np
import pytest

from cases import CASES
from test_smoke_gpu import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 4, 5, 15, 16, 17, 33, 129])
def test_mixed_groups(gpu, count):
    from flowcraft_b200.smoke import SmokeTrailSystem
    from oracle.smoke_oracle import advect
    s, solid = _solver(CASES["sphere48_q19"])
    s.Step(None, 20)
    field = s.ReadbackField()
    nz, ny, nx = solid.shape
    rng = np.random.default_rng(count)
    # world x is grid y, world y is grid x; a margin outside the grid too
    pos = (rng.uniform(-0.1, 1.1, (count, 3)) * np.array([ny, nx, nz])).astype(np.float32)
    steps, length = 3, 6
    sm = SmokeTrailSystem(s)
    sm.Reset(False, count, length)
    sm.SetPositions(pos)
    for _ in range(steps):
        sm.Step(False, 40.0, 1.0 / 60.0, True)  # respawning suspended: the others vanish
    got, lens = sm.Trails()
    cell = np.floor(pos[:, [1, 0, 2]]).astype(int)
    inside = ((cell >= 0) & (cell < [nx, ny, nz])).all(1)
    fluid = inside.copy()
    fluid[inside] = solid[cell[inside, 2], cell[inside, 1], cell[inside, 0]] == 0
    assert (lens[~fluid] == 0).all()
    alone = SmokeTrailSystem(s)
    for p in np.nonzero(fluid)[0]:
        alone.Reset(False, 1, length)
        alone.SetPositions(pos[p:p + 1])
        for _ in range(steps):
            alone.Step(False, 40.0, 1.0 / 60.0, True)
        one, one_len = alone.Trails()
        assert one_len[0] == lens[p]
        assert np.array_equal(one[0].view(np.uint32), got[p].view(np.uint32))
        # the restatement covers the steps up to the one that leaves or vanishes
    keep = fluid & (lens == steps + 1)
    if keep.any():
        want = advect(field, solid, (nx, ny, nz), 1.0, (0.0, 0.0, 0.0), pos[keep], steps, 40.0, 1.0 / 60.0)
        want = want[0] if isinstance(want, tuple) else want
        want = np.asarray(want, np.float32).reshape(keep.sum(), -1, 3)
        assert np.array_equal(got[keep][:, :steps + 1].view(np.uint32), want[:, :steps + 1].view(np.uint32))
    s.close()
