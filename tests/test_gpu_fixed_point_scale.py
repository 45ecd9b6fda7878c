"""The common scale of the fixed-point transforms on vectors that are neither
flat nor a single value (a few peaks on noise, as the brackets of an
intermittent field are), at the sizes of every stage schedule; and the passes'
own conversions far from ordinary magnitudes.

Tolerances: a transform's relative L2 error is at most that of the same
transform in FP64 arithmetic (numpy's, of the same vector).  A power of two in
the state is exact: it changes no bit of a mantissa anywhere in a step.
"""
import numpy as np
import pytest

from tests._helpers import params, random_state

pytestmark = pytest.mark.gpu


def vectors(n):
    rng = np.random.default_rng(n)
    w = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    out = {}
    for peak in (10, 40, 80, 640):
        z = w.copy()
        z[rng.integers(n)] += peak * (1 - 0.5j)
        out["noise and a peak of %d" % peak] = z
    z = w.copy()
    z[rng.integers(0, n, 8)] *= 30
    out["eight peaks"] = z
    out["cubed noise"] = w * np.abs(w) ** 2
    return out


def rel(a, b):
    return float(np.sqrt((np.abs(a - b) ** 2).sum() / (np.abs(b) ** 2).sum()))


@pytest.mark.parametrize("n", [512, 1024, 2048, 4096, 8192])
def test_peaked_vectors_as_exact_as_fp64_arithmetic(gpu, n):
    fwd, inv = gpu.FFTPlan(n, gpu.R2C), gpu.FFTPlan(n, gpu.C2R)
    r, c = np.zeros((n, n)), np.zeros((n // 2 + 1, n), np.complex128)
    for name, z in vectors(n).items():
        # one row: its transform in every column
        r[0] = z.real
        exact = np.fft.rfft(z.real.astype(np.longdouble))
        assert rel(fwd.r2c(r)[:, 0], exact) <= rel(np.fft.rfft(z.real), exact), name
        # column kx = 1: its transform t in the row of every y as 2 Re(t exp(2 pi i x / n))
        c[1] = z
        t = inv.c2r(c)
        exact = np.fft.ifft(z.astype(np.clongdouble)) * n
        assert rel((t[:, 0] - 1j * t[:, n // 4]) / 2, exact) <= rel(np.fft.ifft(z) * n, exact), name


@pytest.mark.parametrize("n,variant", [(32, "per_row_pair"), (256, "per_row_pair"), (256, "split"),
                                       (1024, "per_row_pair")])
def test_step_commutes_with_powers_of_two(gpu, monkeypatch, n, variant):
    monkeypatch.setenv("R2D3C_PASSB", variant)
    _, cp = params(n, omega=0.0, nu=0.0, nuv=0.0, hnu=0.0, hnuv=0.0, iflow=0)
    _, ps, vz = random_state(n, 71, amp=float(n) ** 2)

    def step(a, b):  # psi 2^a, vz 2^b, dt 2^-a: the brackets scale by 2^(2a), 2^(a+b)
        c = gpu.Context(cp, 0)
        c.set_state(ps * 2.0 ** a, vz * 2.0 ** b)
        c.set_forcing(np.zeros_like(ps), np.zeros_like(ps))
        c.step(1e-3 * 2.0 ** -a)
        p, v = c.get_state()
        c.destroy()
        return p * 2.0 ** -a, v * 2.0 ** -b

    p0, v0 = step(0, 0)
    assert np.any(p0 != ps) and np.any(v0 != vz)
    for a, b in ((66, -66), (-66, 66), (0, 300), (0, -300), (300, 300), (-300, -300), (400, -400)):
        p, v = step(a, b)
        np.testing.assert_array_equal(p, p0)
        np.testing.assert_array_equal(v, v0)
