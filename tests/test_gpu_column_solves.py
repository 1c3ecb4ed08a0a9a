"""The column solves on grids on both sides of the lines between their two forms (tiles of columns in shared memory, or a
thread per real or imaginary part), with and without variable-resolution bands, against the oracle."""
import pytest

from tests.helpers import SMALL, projected_ic, rel_l2

pytestmark = pytest.mark.gpu

# columns: 2112 (both solves in tiles), 4704 (the pressure solve), 5940 (neither)
GRIDS = {"both": 96, "pressure": 144, "neither": 162}


@pytest.mark.parametrize("banded", [False, True], ids=["one", "bands"])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_column_solves_against_the_oracle(oracle_mod, grid, banded):
    """Velocity solve, flow rate and pressure correction of one substage, to the tolerance of the substage comparisons,
    and the projection of the field they leave."""
    import littleharsh_gb300 as lh
    n = GRIDS[grid]
    cfg = dict(SMALL, ngalx=n, ngalz=n, ntilex=6, ntilez=6)
    if banded:
        cfg.update(ngalx2=54, ngalz2=72)
    o = oracle_mod.Oracle(**cfg)
    f = projected_ic(o, seed=6)
    dt = o.cfl_dt(0.5)
    o.set_fields(*f)
    o.set_scalars(0.0, dt, 0.0, o.flowrate())
    s = lh.Solver(lh.Config(**cfg))
    s.set_fields(*f)
    s.set_time(0.0, dt, 0.0)
    for upto in (3, 5):
        o.substage(1, upto)
        s.substage(1, upto)
        for a, b in zip(s.get_fields(), o.get_fields()):
            assert rel_l2(a, b) < 1e-11
    s.step(2)
    o.step(2)
    for a, b in zip(s.get_fields(), o.get_fields()):
        assert rel_l2(a, b) < 1e-10
    assert s.divmax() < 1e-12
    u = s.get_fields()
    s.project()  # last: it takes the target flow rate from the field
    for a, b in zip(s.get_fields(), u):
        assert rel_l2(a, b) < 1e-11
