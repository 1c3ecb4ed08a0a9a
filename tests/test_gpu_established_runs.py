"""FP64 runs come out as they always have: the plane mean of v, a zero by continuity that holds nothing but the step's
roundings, and the CFL time step after a few steps are compared with recorded ones."""
import json
import os

import numpy as np
import pytest

from tests.helpers import SMALL

pytestmark = pytest.mark.gpu

RECORDED = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "established_fp64.json")
# canopy: 40 pressure levels; bands: lower bands of 15; three43: 43, three beyond the last whole four; three43_columns: the
# same with too many columns for tiles; ragged: 48
RUNS = {"canopy": SMALL, "bands": dict(SMALL, ngalx2=18, ngalz2=18), "three43": dict(SMALL, ny=36),
        "three43_columns": dict(SMALL, ny=36, ngalx=288, ngalz=96, ntilex=12, ntilez=6),
        "ragged": dict(SMALL, ngalx=54, ngalz=36, ny=41, ntilex=9, ntilez=6, flag_ctpress=1)}


def _fields(s, kept):
    """A perturbed parabola from integers and IEEE products and sums alone: the same bits on every host."""
    rng = np.random.default_rng(7)
    out = []
    for y, scale in ((s.grid["yu"], 2.0**-14), (s.grid["yv"], 2.0**-14), (s.grid["yu"], 2.0**-14), (s.grid["yu"][1:-1], 2.0**-16)):
        f = np.zeros((y.size, s.nz, s.nkx), np.complex128)
        env = np.maximum(1.0 - y * y, 0.0)
        for part in (f.real, f.imag):
            c = np.zeros((s.nz, s.nkx))
            c[-kept:, 1:kept] = scale * rng.integers(-256, 257, (kept, kept - 1))
            c[:kept, 1:kept] = scale * rng.integers(-256, 257, (kept, kept - 1))
            part[:] = env[:, None, None] * c
        out.append(f)
    y = s.grid["yu"]
    out[0][:, 0, 0] = 1.5 * np.maximum(1.0 - y * y, 0.0)
    return out


def run(lh, cfg):
    """Two output intervals of two steps: {quantity: values}."""
    s = lh.Solver(lh.Config(**cfg))
    s.set_fields(*_fields(s, 5))
    s.set_time(0.0, 1.0, -0.004 if cfg["flag_ctpress"] else 0.0)
    s.project()
    s.set_time(0.0, 2.0**-8, s.time()["mpgx"])
    out = {"dt": [], "mpgx": []}
    for _ in range(2):
        s.step(2)
        s.stats_accumulate()
        now = s.time()
        s.set_time(now["t"], s.cfl_dt(0.5), now["mpgx"])
        out["dt"].append(s.time()["dt"])
        out["mpgx"].append(now["mpgx"])
    out["Vm"] = [float(x) for x in s.stats_flush()[1]["Vm"]]
    s.close()
    return out


@pytest.mark.parametrize("name", list(RUNS))
def test_established_run(name):
    """Each quantity to 1e-9 of its norm, the bound of an FP64 output: the plane mean of v keeps it only if the roundings
    are the same throughout."""
    import littleharsh_gb300 as lh
    with open(RECORDED) as f:
        want = json.load(f)[name]
    got = run(lh, RUNS[name])
    for k, v in want.items():
        a, b = np.array(got[k]), np.array([float.fromhex(x) for x in v])
        assert a.shape == b.shape and np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b), k


@pytest.mark.parametrize("cfg", [SMALL, dict(SMALL, ngalx=288, ngalz=96, ntilex=12, ntilez=6)], ids=["tiles", "columns"])
def test_right_hand_sides_after_the_velocity_solves(cfg):
    """After the velocity solves the right-hand sides hold the forward sweep, whichever form a grid's solves take: the last
    level of each is the velocity there, bit for bit."""
    import littleharsh_gb300 as lh
    s = lh.Solver(lh.Config(**cfg))
    s.set_fields(*_fields(s, 5))
    s.set_time(0.0, 1.0, 0.0)
    s.project()
    s.set_time(0.0, 2.0**-8, 0.0)
    s.substage(1, 3)
    for r, u in zip(s.get_rhs(), s.get_fields()):
        np.testing.assert_array_equal(r[-1], u[-1])
    assert s.get_rhs()[0][-1].any()
