"""The FP64 transforms in 64-bit fixed point: their error against extended precision on the CPU, and the step's
passes at the lengths where they differ, on the GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from tests.helpers import SMALL, SMOOTH, projected_ic, rel_l2

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "littleharsh_gb300", "csrc")
# every first, middle and last pass, one part missing, and the lengths in use
LENGTHS = [6, 8, 9, 16, 18, 24, 27, 48, 54, 64, 81, 96, 108, 128, 144, 162, 192, 216, 243, 288, 324, 384, 432, 486, 512,
           576, 768, 972, 1152, 2304]


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    from littleharsh_gb300 import build
    so = str(tmp_path_factory.mktemp("fx") / "fx_host.so")
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I" + CSRC,
                    os.path.join(HERE, "native", "fx_host.cu"), "-o", so], check=True, capture_output=True)
    lib = C.CDLL(so)

    def run(x, inverse):
        x = np.ascontiguousarray(x, np.complex128)
        out = np.empty_like(x)
        assert lib.fx_host(x.size, int(inverse), x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
        return out
    return run


def _exact(x, inverse):
    x = x.astype(np.clongdouble)
    return np.fft.ifft(x) * x.size if inverse else np.fft.fft(x)


def _lines(n, rng):
    """(inverse, line): spectra (flat, falling off, one large mode, a single mode) and physical lines (noise, noise on a
    mean, smooth on a mean)."""
    k = np.minimum(np.arange(n), n - np.arange(n))
    c = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    kept = k < max(n // 3, 2)
    falling = c * (1 + k**2 / 36) ** (-4 / 3) * kept
    mean = 0.02 * falling
    mean[0] = 1.0
    one = np.zeros(n, complex)
    one[n // 3] = 0.7 + 0.2j
    smooth = np.fft.ifft(falling * (k > 0)) * n + 3
    return [(1, c * kept), (1, falling), (1, mean), (1, one), (0, c), (0, 1 + 0.1 * c), (0, smooth)]


@pytest.mark.parametrize("n", LENGTHS)
def test_error_is_no_larger_than_fp64(host, n):
    """2-norm error against extended precision, mean of eight lines of a kind: at most that of an FP64 FFT of the same
    lines, or one FP64 unit roundoff where FP64 happens to be exact."""
    rng = np.random.default_rng(n)
    err = np.zeros((7, 2))
    for _ in range(8):
        for i, (inv, x) in enumerate(_lines(n, rng)):
            ref = _exact(x, inv)
            fp64 = np.fft.ifft(x) * n if inv else np.fft.fft(x)
            scale = np.linalg.norm(ref)
            err[i] += [np.linalg.norm(host(x, inv) - ref) / scale, np.linalg.norm(fp64 - ref) / scale]
    err /= 8
    assert np.all(err[:, 0] <= np.maximum(err[:, 1], 2.0**-53)), err * 2.0**53


@pytest.mark.parametrize("n", [9, 54, 96, 486, 576, 1152])
def test_largest_lines_do_not_overflow(host, n):
    """Lines whose parts are all as large as a line's largest, signed so that one frequency adds them all up (the bound of
    a forward line), and spectra that add up in one point (the bound of an inverse one)."""
    rng = np.random.default_rng(3)
    s = np.arange(n)
    for q in {1, n // 3, n // 2, n - 1, int(rng.integers(n))}:
        w = np.exp(2j * np.pi * s * q / n)
        big = np.where(w.real >= 0, 1.0, -1.0) + 1j * np.where(w.imag >= 0, 1.0, -1.0)
        big *= np.nextafter(1.0, 0.0)
        for inv in (0, 1):
            ref = _exact(big, inv)
            assert np.linalg.norm(host(big, inv) - ref) < 8 * 2.0**-53 * np.linalg.norm(ref)


@pytest.mark.parametrize("scale", [1e-300, 1e-30, 1e30, 1e150])
def test_scale_of_a_line_does_not_matter(host, scale):
    """A power of two of a line is the same integers."""
    rng = np.random.default_rng(4)
    x = rng.standard_normal(96) + 1j * rng.standard_normal(96)
    two = 2.0 ** np.floor(np.log2(scale))
    for inv in (0, 1):
        np.testing.assert_array_equal(host(x * two, inv), host(x, inv) * two)
    assert not host(np.zeros(96), 1).any()


# z lengths: powers of two and of three alone, 2 and 4 as the first radix, 3 and 9 as the last, twiddled passes of each
Z_LENGTHS = [6, 8, 9, 16, 18, 27, 32, 54, 64, 81, 108, 128, 162]


# x lengths (even): the same, and one beyond two levels per iteration of the product pass
X_LENGTHS = [6, 8, 16, 18, 32, 54, 64, 128, 162, 486, 1944]


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [dict(SMOOTH, ngalz=n) for n in Z_LENGTHS] + [dict(SMOOTH, ngalx=n, ngalz=12) for n in X_LENGTHS],
                         ids=[f"z{n}" for n in Z_LENGTHS] + [f"x{n}" for n in X_LENGTHS])
def test_lengths_against_the_oracle(oracle_mod, cfg):
    """Right-hand sides and nonlinear term of the first substage, to the tolerance of the other substage comparisons, and
    the CFL time step."""
    import littleharsh_gb300 as lh
    o = oracle_mod.Oracle(**cfg)
    f = projected_ic(o, seed=2)
    dt = o.cfl_dt(0.5)
    o.set_fields(*f)
    o.set_scalars(0.0, dt, 0.0, o.flowrate())
    s = lh.Solver(lh.Config(**cfg))
    s.set_fields(*f)
    s.set_time(0.0, dt, 0.0)
    o.substage(1, 1)
    s.substage(1, 1)
    for a, b in zip(s.get_nonlinear() + s.get_rhs(), list(o.get_nonlinear()) + list(o.get_rhs())):
        assert rel_l2(a, b) < 1e-11
    assert abs(s.cfl_dt(0.5) - o.cfl_dt(0.5)) < 1e-12 * dt


# canopy rows in pairs: an odd row left over, pairs with one or no solid row, one post, lines of one and of several warps
CANOPY = [dict(ngalx=16, ngalz=9, ntilex=2, ntilez=1, dstx=1, dstz=1), dict(ngalx=54, ngalz=27, ntilex=3, ntilez=3, dstx=5, dstz=2),
          dict(ngalx=128, ngalz=16, ntilex=1, ntilez=1, dstx=1, dstz=1), dict(ngalx=486, ngalz=18, ntilex=6, ntilez=2),
          dict(ngalx=1152, ngalz=12, ntilex=4, ntilez=4)]


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [dict(SMALL, **c) for c in CANOPY], ids=[f"{c['ngalx']}x{c['ngalz']}" for c in CANOPY])
def test_canopy_rows_against_the_oracle(oracle_mod, cfg):
    """Right-hand sides after the canopy forcing of the first substage, to the tolerance of the other substage comparisons."""
    import littleharsh_gb300 as lh
    o = oracle_mod.Oracle(**cfg)
    f = projected_ic(o, seed=3)
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


@pytest.mark.gpu
def test_zero_lines_stay_zero():
    """A field of zeros has a nonlinear term of exact zeros, and rows without a velocity component do not disturb others."""
    import littleharsh_gb300 as lh
    s = lh.Solver(lh.Config(**SMALL))
    f = s.get_fields()
    s.set_fields(*[np.zeros_like(x) for x in f])
    s.set_time(0.0, 1e-3, 0.0)
    s.substage(1, 1)
    for n in s.get_nonlinear():
        assert not n.any()
    u = np.zeros_like(f[0])
    u[:, 0, 0] = np.linspace(1.0, 2.0, u.shape[0])
    s.set_fields(u, np.zeros_like(f[1]), np.zeros_like(f[2]), np.zeros_like(f[3]))
    s.substage(1, 1)
    for n in s.get_nonlinear():  # d/dx, d/dz of u(y)^2 and d/dy of products with v = 0
        assert np.abs(n).max() < 1e-14


@pytest.mark.gpu
@pytest.mark.parametrize("banded", [False, True], ids=["one", "bands"])
def test_chunks_of_levels_keep_results(monkeypatch, banded):
    """Chunks of one, three and any number of levels start at whole pairs of levels: bit for bit the same step."""
    import littleharsh_gb300 as lh
    from littleharsh_gb300.initial import initial_field
    cfg = dict(SMALL, ngalx2=18, ngalz2=18) if banded else SMALL
    ref = None
    for chunk in ("64", "1", "3", "6"):
        monkeypatch.setenv("LH_CHUNK", chunk)
        s = lh.Solver(lh.Config(**cfg))
        g = s.grid
        s.set_fields(*initial_field(g["yu"], g["yv"], s.nz, s.nkx, s.nyp, seed=9, kmax=4))
        s.project()
        s.set_time(0.0, 1e-3, 0.0)
        s.step(2)
        f = s.get_fields()
        assert all(np.all(np.isfinite(x)) for x in f)
        if ref is not None:
            for a, b in zip(f, ref):
                np.testing.assert_array_equal(a, b)
        ref = f
