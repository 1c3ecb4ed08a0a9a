"""Planes with an odd number of values."""
import numpy as np
import pytest

from tests.helpers import SMALL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ngalz", [24, 27])
def test_conditional_statistics_of_the_mixed_form(ngalz):
    """Conditional statistics read the FP64 fields in either form, through FP64 planes in the step's buffers: the same bits
    from both.  With Ngalz = 27 a plane holds 13 x 27 values and a face field 41 planes, so that the mixed form's buffers
    have odd sizes."""
    import littleharsh_gb300 as lh
    cfg = dict(SMALL, ngalx=36, ntilex=6, ngalz=ngalz, ntilez=3)
    rng = np.random.default_rng(4)
    sums, f = [], None
    for prec in (lh.PREC_FP64, lh.PREC_MIXED):
        s = lh.Solver(lh.Config(**cfg), precision=prec)
        if f is None:
            f = []
            for x in s.get_fields():
                x = np.zeros_like(x)
                x[:, :, 1:] = rng.standard_normal(x[:, :, 1:].shape) + 1j * rng.standard_normal(x[:, :, 1:].shape)
                x[:, 0, 0] = 1.0
                f.append(x)
        s.set_fields(*f)
        s.cond_accumulate()
        sums.append(s.cond_flush()[1])
        s.set_time(0.0, 1e-4, 0.0)
        s.step(1)
        assert all(np.isfinite(x).all() for x in s.get_fields())
    for k, v in sums[0].items():
        np.testing.assert_array_equal(v, sums[1][k])
