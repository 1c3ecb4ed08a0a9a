"""Column solves of grids with thousands of levels."""
import numpy as np
import pytest

from tests.helpers import SMOOTH

pytestmark = pytest.mark.gpu


def _solver(cfg):
    import littleharsh_gb300 as lh
    s = lh.Solver(lh.Config(**cfg))
    rng = np.random.default_rng(6)
    y = {"u": s.grid["yu"], "v": s.grid["yv"]}
    f = [np.zeros_like(x) for x in s.get_fields()]
    for x, g in zip(f[:3], "uvu"):
        env = np.maximum(1.0 - y[g] ** 2, 0.0) ** 2
        x[:, 1, 1:2] = env[:, None] * (0.01 * rng.standard_normal() + 0.01j * rng.standard_normal())
    f[0][:, 0, 0] = np.maximum(1.0 - y["u"] ** 2, 0.0)
    s.set_fields(*f)
    s.set_time(0.0, 1.0, 0.0)
    return s


@pytest.mark.parametrize("ny", [6142, 6143, 6145, 9001])
def test_projection_and_step_beyond_6144_faces(ny):
    """A column's factors fit 48 KB of shared memory to 6144 faces; beyond that they are read from global memory.  The
    projection removes the divergence (the field's is about 0.02) and a step runs, alone and in a batched launch."""
    import littleharsh_gb300 as lh
    cfg = dict(SMOOTH, ngalx=6, ngalz=6, ny=ny)
    s, a, b = (_solver(cfg) for _ in range(3))
    before = s.divmax()
    assert before > 1e-3
    for q in (s, a, b):
        q.project()
        q.set_time(0.0, 1e-7, 0.0)
    assert s.divmax() < 1e-6 * before
    s.step(1)
    e = lh.Ensemble([a, b], mode=lh.ENS_BATCHED)
    e.step(1)
    for x, y, z in zip(s.get_fields(), a.get_fields(), b.get_fields()):
        assert np.isfinite(x).all()
        np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(x, z)
