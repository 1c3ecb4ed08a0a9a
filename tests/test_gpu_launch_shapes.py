"""Launch shapes at the limits of shared memory and of the rules that choose them."""
import numpy as np
import pytest

from tests.helpers import C1, SMALL, SMOOTH, projected_ic, rel_l2

pytestmark = pytest.mark.gpu


def _stepped(cfg, precision, tune=False):
    import littleharsh_gb300 as lh
    s = lh.Solver(lh.Config(**cfg), precision=precision)
    rng = np.random.default_rng(5)
    f = [np.zeros_like(x) for x in s.get_fields()]
    for x in f[:3]:
        n = min(8, x.shape[2] - 1)
        x[1:-1, 1:3, 1:n + 1] = 0.01 * rng.standard_normal((x.shape[0] - 2, 2, n))
    f[0][:, 0, 0] = 1.0
    s.set_fields(*f)
    s.set_time(0.0, 1.0, 0.0)
    s.project()
    s.set_time(0.0, 1e-4, 0.0)
    if tune:
        s.autotune()
    s.step(1)
    return s.launch_shapes(), s.get_fields()


@pytest.mark.parametrize("n,rows", [(2304, 2), (2592, 1), (4374, 1)])
def test_mixed_product_pass_takes_two_rows_where_they_fit(monkeypatch, n, rows):
    """Two z rows per CTA want about 99 bytes of shared memory a point of x: they fit at 2304, not at 2592, and the one-row
    kernel serves on; the same bits either way, tuned or not."""
    import littleharsh_gb300 as lh
    cfg = dict(SMOOTH, ngalx=n, ngalz=6, ny=13)
    shapes, f = _stepped(cfg, lh.PREC_MIXED)
    assert shapes["xrows"] == rows
    assert all(np.isfinite(x).all() for x in f) and np.abs(f[0]).max() > 0.5
    tuned, g = _stepped(cfg, lh.PREC_MIXED, tune=True)
    assert tuned["xrows"] <= rows
    monkeypatch.setenv("LH_XROWS", "1")
    _, one = _stepped(cfg, lh.PREC_MIXED)
    for a, b, c in zip(f, g, one):
        np.testing.assert_array_equal(a, c)
        np.testing.assert_array_equal(b, c)


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_tuning_tries_what_the_rule_takes(mixed):
    """The default chunk of levels is one that the tuner times.  Half of configuration 1 in the mixed form takes two levels,
    40 % faster than four, which the tuner has to find as well."""
    import littleharsh_gb300 as lh
    prec = lh.PREC_MIXED if mixed else lh.PREC_FP64
    cfg = dict(C1, ngalx=48, ngalz=48, ny=49, dsty=8, dstx=1, dstz=2)
    default, f = _stepped(cfg, prec)
    assert default["chunk"] == (2 if mixed else 4)
    tuned, g = _stepped(cfg, prec, tune=True)
    assert tuned["chunk"] in ((2,) if mixed else (4, 8, 16, 32, 64))
    for a, b in zip(f, g):
        np.testing.assert_array_equal(a, b)


def test_canopy_forcing_on_the_shortest_rows(oracle_mod):
    """Ngalx = 6 with posts: right-hand sides after the canopy forcing, to the tolerance of the other substage
    comparisons."""
    import littleharsh_gb300 as lh
    cfg = dict(SMALL, ngalx=6, ngalz=12, ntilex=2, ntilez=3, dstx=1, dstz=2)
    o = oracle_mod.Oracle(**cfg)
    f = projected_ic(o, seed=3, kmax=2)
    dt = o.cfl_dt(0.5)
    o.set_fields(*f)
    o.set_scalars(0.0, dt, 0.0, o.flowrate())
    s = lh.Solver(lh.Config(**cfg))
    s.set_fields(*f)
    s.set_time(0.0, dt, 0.0)
    o.substage(1, 2)
    s.substage(1, 2)
    for a, b in zip(s.get_rhs(), o.get_rhs()):
        assert rel_l2(a, b) < 1e-11


def test_tuned_mixed_planes_beyond_the_fixed_point_tables():
    """The mixed form takes z lengths that the FP64 passes and their tables do not reach, with the tile width that the tuner
    finds to fit."""
    import littleharsh_gb300 as lh
    shapes, f = _stepped(dict(SMOOTH, ngalx=6, ngalz=18432, ny=13), lh.PREC_MIXED, tune=True)
    assert shapes["tx"] == 1
    assert all(np.isfinite(x).all() for x in f) and np.abs(f[0]).max() > 0.5
