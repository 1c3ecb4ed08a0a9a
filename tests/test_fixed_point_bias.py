"""The fixed-point transforms have no error of one sign, keep exact zeros, and take lines of any scale."""
import numpy as np
import pytest

from tests.helpers import SMALL
from tests.test_fixed_point_fft import _exact, host  # noqa: F401


@pytest.mark.parametrize("n", [54, 96, 162, 288, 576])
@pytest.mark.parametrize("kind", ["falling", "flat", "physical"])
def test_errors_have_no_mean(host, n, kind):  # noqa: F811
    """Over 60 lines: at every output the mean error is within an FP64 unit roundoff of the lines' rms, and the largest
    error is no larger than that of FP64 transforms."""
    rng = np.random.default_rng(n)
    k = np.minimum(np.arange(n), n - np.arange(n))
    kept = k < n // 3
    err, fp64 = [], []
    for _ in range(60):
        c = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        x = {"falling": c * (1 + k**2 / 36) ** (-4 / 3) * kept, "flat": c * kept, "physical": 1 + 0.1 * c}[kind]
        inv = kind != "physical"
        ref = _exact(x, inv)
        rms = np.sqrt(np.mean(np.abs(ref) ** 2))
        err.append(((host(x, inv) - ref) / rms).astype(complex))
        fp64.append((((np.fft.ifft(x) * n if inv else np.fft.fft(x)) - ref) / rms).astype(complex))
    mean = np.mean(err, 0)
    assert max(np.abs(mean.real).max(), np.abs(mean.imag).max()) <= 2.0**-53
    largest = [max(np.abs(np.real(e)).max(), np.abs(np.imag(e)).max()) for e in (err, fp64)]
    assert largest[0] <= largest[1]


@pytest.mark.parametrize("n", [16, 27, 96, 162, 576])
def test_zeros_stay_zeros(host, n):  # noqa: F811
    """A constant line has one frequency and a single mean mode one value at every point: what cancels exactly is zero."""
    out = host(np.full(n, 0.7 - 0.3j), 0)
    assert np.count_nonzero(out) == 1 and abs(out[0] - n * (0.7 - 0.3j)) <= 2.0**-51 * n
    x = np.zeros(n, complex)
    x[0] = 0.7 - 0.3j
    assert np.all(host(x, 1) == x[0])


@pytest.mark.gpu
@pytest.mark.parametrize("power", [-900, -600, 600, 900])
def test_conditional_sums_of_any_scale(power):
    """The linear conditional sums of a field times a power of two are theirs times that power: lines near the ends of
    FP64's range are scaled by other instructions, and so are values far below their line's largest.  The modes are those
    that a sum over the 4 x 4 tiles keeps."""
    import littleharsh_gb300 as lh
    rng = np.random.default_rng(8)
    s = lh.Solver(lh.Config(**SMALL))
    f = []
    for x in s.get_fields():
        x = np.zeros_like(x)
        for kx, kz, scale in ((4, 0, 1.0), (4, 4, 0.5), (8, -4, 0.25), (4, -4, 2.0**-90)):
            x[:, kz, kx] = scale * (rng.standard_normal(x.shape[0]) + 1j * rng.standard_normal(x.shape[0]))
        x[:, 0, 0] = 1.0
        f.append(x)
    sums = []
    for p in (0, power):
        s.set_fields(*[x * 2.0**p for x in f])
        s.cond_accumulate()
        sums.append(s.cond_flush()[1])
    for name, x in zip(("UmC", "VmC", "WmC", "PmC"), f):
        a, b = sums[0][name], sums[1][name] * 2.0 ** (-power)
        # 32 values a sum (16 tiles, two walls), each of two runs within eight roundings of the moduli's sum
        most = 2 * np.abs(x).sum((1, 2)).max()
        assert np.isfinite(b).all() and np.abs(a).max() > most and np.abs(a - b).max() <= 32 * 2 * 8 * 2.0**-53 * most, name
