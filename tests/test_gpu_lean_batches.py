"""FP32 pass B at n = 2048 in batches (an odd number of runs, so that the
persistent CTAs of a run do not divide its row pairs evenly): each schedule
forced, against single runs under the other one.  Bit for bit: a row pair is
computed the same way whatever CTA carries it."""
import numpy as np
import pytest

from tests._helpers import params, random_forcing, random_state

pytestmark = pytest.mark.gpu


def test_batches_under_either_schedule(gpu, monkeypatch):
    n, runs = 2048, []
    for i in range(3):
        _, cp = params(n, omega=1.0 + i, nu=1e-5, nuv=1e-5, hnu=0.1, hnuv=0.1, iflow=0)
        g, ps, vz = random_state(n, 90 + i, kmax_shell=100.0, slope=-3.0, amp=float(n) ** 2)
        runs.append((cp, ps, vz, *random_forcing(g, 95 + i, 20.0, 22.0)))
    for batch, single in (("persistent", "per_row_pair"), ("per_row_pair", "persistent")):
        monkeypatch.setenv("R2D3C_PASSB", batch)
        ens = gpu.Ensemble([(n, [r[0] for r in runs])], gpu.FP32)
        assert ens.plan_report()[0]["plan"]["chosen"] == batch
        for i, (_, ps, vz, fp, fz) in enumerate(runs):
            ens.set_state(i, ps, vz)
            ens.set_forcing(i, fp, fz)
            ens.set_time(i, 0.0)
        times = ens.advance(2, gpu.DT_CFL, 0.5)
        monkeypatch.setenv("R2D3C_PASSB", single)
        for i, (cp, ps, vz, fp, fz) in enumerate(runs):
            c = gpu.Context(cp, gpu.FP32)
            assert c.plan_report()["chosen"] == single
            c.set_state(ps, vz)
            c.set_forcing(fp, fz)
            c.set_time(0.0)
            assert c.advance(2, gpu.DT_CFL, 0.5)[0] == times[i]
            for a, b in zip(c.get_state(), ens.get_state(i)):
                np.testing.assert_array_equal(a, b)
            c.destroy()
        ens.destroy()
