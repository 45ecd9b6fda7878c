"""The maxima that a pass takes over its lanes (the CFL time step; the field
extrema of the diagnostics) on grids whose blocks hold fewer threads than a
warp: every launch shape against the oracle, a strong state before a weak one,
so that a value left in a lane that does not exist would be the larger one.

Tolerance: a velocity is a sum over the modes through two passes of log2 n
stages of rounding 2^-53 (2^-24 in FP32, whose squares double it); 32 such
roundings a stage cover the largest of n^2 values.
"""
import numpy as np
import pytest

from oracle import rot2d3c_oracle as O
from tests._helpers import params, random_forcing, random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_time_step_and_extrema(gpu, monkeypatch, n, prec):
    tol = 2.0 ** (-53 if prec == 0 else -24) * 32 * np.log2(n)
    p, cp = params(n, omega=1.0, cfl=0.4, nu=1e-4, nuv=1e-4, iflow=0)
    for variant, groups in (("per_row_pair", "1,1,1,1"), ("per_row_pair", "0,1,0,0"), ("split", "0,1,0,0"),
                            ("per_row_pair", "2,1,2,2")):
        monkeypatch.setenv("R2D3C_PASSB", variant)
        monkeypatch.setenv("R2D3C_GROUPS", groups)
        for amp in (1e4, 1.0):
            g, ps, vz = random_state(n, 61, amp=amp * n ** 2)
            fp, fz = random_forcing(g, 62, 2.0, 4.0)
            c = gpu.Context(cp, prec)
            assert c.plan_report()["chosen"] == variant
            c.set_state(ps, vz)
            c.set_forcing(fp, fz)
            c.set_time(0.0)
            want = O.cond_check(g, p, ps, vz, fp, fz, 0.0)[-4:]
            got = c.cond_check(0.0)[-4:]
            assert np.all(np.abs(got - want) <= tol * np.abs(want).max()), (variant, groups, amp)
            dt = O.cfl_condition(g, p, ps, vz)
            assert abs(c.advance(1, gpu.DT_CFL, p.cfl)[1] - dt) <= tol * dt, (variant, groups, amp)
            c.destroy()
