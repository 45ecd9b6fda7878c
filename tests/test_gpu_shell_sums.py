"""Shell and half-plane sums at the grids' ends: the smallest grids (shells of
a few elements, the kx = n/2 and ky = -n/2 lines), and a full plane of random
values in which every element counts, against the oracle.

Tolerance: FP64 sums of up to n^2 terms of both signs in another order;
relative to the sum of magnitudes 2^-53 * log2(n^2) + the terms' own roundings:
below 1e-14.
"""
import numpy as np
import pytest

from oracle import rot2d3c_oracle as O
from tests._helpers import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 64, 256, 1024])
@pytest.mark.parametrize("mm,nn", [(2, 1), (0, 4), (3, 2)])
def test_full_plane(gpu, n, mm, nn):
    p, cp = params(n, omega=1.3, nu=1e-3, nuv=2e-3, hnu=0.1, hnuv=0.2, nn=nn, mm=mm, nnv=nn, mmv=mm, kup=3.0, iflow=0)
    g = O.Grid(n)
    rng = np.random.default_rng(n + mm)
    ps, vz, fp, fz = (rng.standard_normal((n // 2 + 1, n)) + 1j * rng.standard_normal((n // 2 + 1, n))
                      for _ in range(4))
    c = gpu.Context(cp, 0)
    c.set_state(ps, vz)
    c.set_forcing(fp, fz)
    ek, ezk = c.spectrum()
    kmn = O.shell_index(g)
    nb = n // 2 + 1
    ok = (kmn > 0) & (kmn <= nb)
    for got, w in ((ek, g.two * g.ka2 * np.abs(ps) ** 2), (ezk, g.two * np.abs(vz) ** 2)):
        ref = np.bincount(np.where(ok, kmn - 1, 0).ravel(), weights=np.where(ok, w, 0.0).ravel(), minlength=nb)[:nb]
        np.testing.assert_allclose(got, ref / g.nrm4, rtol=1e-14)
    got, ref = c.cond_check(0.5), O.cond_check(g, p, ps, vz, fp, fz, 0.5)
    # the inner products' scale: the root of the two energies
    scale = np.abs(ref)
    for i, (a, b, kin) in {3: (ps, fp, 1), 4: (vz, fz, 0), 14: (ps, fp, 2), 18: (vz, ps, 1), 19: (vz, fp, 1),
                           20: (ps, fz, 1)}.items():
        scale[i] = np.sqrt(O.energy(g, a, kin) * O.energy(g, b, kin))
    scale[9] = 2 * p.omega * np.sqrt(O.energy(g, vz, 0) * O.energy(g, ps, 1))
    for i, (q, kin) in {21: (p.nu, nn + 1), 22: (p.nuv, nn + 1), 23: (p.hnu, 1 - mm), 24: (p.hnuv, 1 - mm)}.items():
        scale[i] = q * np.sqrt(O.energy(g, ps, kin) * O.energy(g, vz, kin))
    assert np.max(np.abs(got - ref)[:25] / np.where(scale > 0, scale, 1.0)[:25]) < 1e-14
