"""The FP64 right-hand-side assembly with one, two and four levels a thread and every number of levels left over, against
the oracle."""
import pytest

from tests.helpers import SMALL, projected_ic, rel_l2

pytestmark = pytest.mark.gpu

# (Ngalx = Ngalz, ny): points of a column grid below 100 000, below a million, above
GRIDS = [(24, 33), (24, 34), (96, 54), (96, 55), (192, 130), (192, 131), (192, 132), (192, 133)]


@pytest.mark.parametrize("banded", [False, True], ids=["one", "bands"])
@pytest.mark.parametrize("n,ny", GRIDS)
def test_assembly_against_the_oracle(oracle_mod, n, ny, banded):
    """Right-hand sides and nonlinear terms of two substages (the second reads the first's nonlinear term), to the tolerance
    of the substage comparisons."""
    import littleharsh_gb300 as lh
    cfg = dict(SMALL, ngalx=n, ngalz=n, ny=ny)
    if banded:
        cfg.update(ngalx2=2 * n // 3, ngalz2=n // 2)
    o = oracle_mod.Oracle(**cfg)
    f = projected_ic(o, seed=8)
    dt = o.cfl_dt(0.5)
    o.set_fields(*f)
    o.set_scalars(0.0, dt, 0.0, o.flowrate())
    s = lh.Solver(lh.Config(**cfg))
    s.set_fields(*f)
    s.set_time(0.0, dt, 0.0)
    for k, upto in ((1, 5), (2, 1)):
        o.substage(k, upto)
        s.substage(k, upto)
    for a, b in zip(s.get_nonlinear() + s.get_rhs(), list(o.get_nonlinear()) + list(o.get_rhs())):
        assert rel_l2(a, b) < 1e-11
