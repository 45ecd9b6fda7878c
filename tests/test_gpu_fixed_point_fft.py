"""The FP64 transforms' fixed-point arithmetic at the ends of its range:
vectors of every kind of spread, scales near both ends of the exponent range,
zero and non-finite vectors, each grid size's stage schedule (against
long-double transforms).

Tolerance: the relative L2 error of a 2-D transform in FP64 arithmetic is
about 0.6 * 2^-53 * sqrt(2 log2 n) (2.2e-16 .. 3e-16); the fixed-point one has
to be below it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def bound(n):
    return 0.6 * 2.0 ** -53 * np.sqrt(2 * np.log2(n)) * 1.5  # 1.5: one draw's spread


def fields(n):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    white = rng.standard_normal((n, n))
    spike = np.zeros((n, n))
    spike[n // 3, n // 5] = 1.0
    return {
        "white": white,
        "spiky": white ** 7,
        "spike": spike,
        "constant": np.full((n, n), 0.1),
        "one_mode": np.cos(2 * np.pi * 3 * i / n)[None, :] * np.sin(2 * np.pi * 5 * i / n + 0.3)[:, None],
        "nyquist": (-1.0) ** i[None, :] * np.ones(n)[:, None],
        "rows_apart": white * 10.0 ** rng.uniform(-30, 30, (n, 1)),
        "columns_apart": white * 10.0 ** rng.uniform(-30, 30, (1, n)),
    }


def r2c(r):
    return np.fft.fft(np.fft.rfft(r.astype(LD), axis=1), axis=0).T


def c2r(c, n):
    t = (np.fft.ifft(c.astype(np.clongdouble), axis=1) * n).T.copy()
    t[:, 0] = t[:, 0].real
    t[:, n // 2] = t[:, n // 2].real
    return np.fft.irfft(t, n=n, axis=1) * n


def rel(a, b):
    return float(np.sqrt((np.abs(a - b) ** 2).sum() / (np.abs(b) ** 2).sum()))


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512])
def test_error_below_fp64_arithmetic(gpu, n):
    f, b = gpu.FFTPlan(n, gpu.R2C), gpu.FFTPlan(n, gpu.C2R)
    for name, x in fields(n).items():
        exact = r2c(x)
        assert rel(f.r2c(x), exact) < bound(n), name
        spec = np.asarray(exact, np.complex128)
        assert rel(b.c2r(spec), c2r(spec, n)) < bound(n), name


@pytest.mark.parametrize("exponent", [-1000, -300, 300, 960])
def test_any_exponent(gpu, exponent):
    n = 64
    x = fields(n)["white"]
    f = gpu.FFTPlan(n, gpu.R2C)
    # a power of two changes nothing but the exponent
    assert np.array_equal(f.r2c(np.ldexp(x, exponent)), f.r2c(x) * 2.0 ** exponent)


def test_subnormal_and_zero(gpu):
    n = 64
    f = gpu.FFTPlan(n, gpu.R2C)
    x = np.ldexp(fields(n)["white"], -1062)
    err = np.abs(np.asarray(f.r2c(x) - r2c(x), np.complex128))
    # one last place of a subnormal per rounding: the row result, then the column sums of n of them
    assert err.max() <= 2.0 ** -1074 * 4 * np.sqrt(n)
    assert not np.any(f.r2c(np.zeros((n, n))))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite(gpu, bad):
    n = 64
    x = fields(n)["white"]
    x[5, 7] = bad
    out = gpu.FFTPlan(n, gpu.R2C).r2c(x)
    assert not np.any(np.isfinite(out.real) & np.isfinite(out.imag))
