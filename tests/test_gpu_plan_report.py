"""The plan report names the launch shapes that run: the one shape of the lean
pass C (FP32, n >= 1024) whatever R2D3C_GROUPS asks for, and the shape of pass C
with the next substep's pass A in it."""
import pytest

from tests._helpers import params

pytestmark = pytest.mark.gpu


def _report(gpu, n):
    c = gpu.Context(params(n, iflow=0)[1], gpu.FP32)
    rep = c.plan_report()
    c.destroy()
    return rep


def test_lean_pass_c_shape(gpu, monkeypatch):
    monkeypatch.setenv("R2D3C_PASSC", "per_column_pair")
    for groups in ("0,1,1,1,1", "0,1,2,2,2,2", "0,1,0,0", None):
        if groups:
            monkeypatch.setenv("R2D3C_GROUPS", groups)
        else:
            monkeypatch.delenv("R2D3C_GROUPS")
        rep = _report(gpu, 1024)
        assert (rep["groups_c"], rep["chunks_c"], rep["team_c"]) == (1, 2, 1), groups
        shapes = [(r["groups"], r["chunks"], r["team"]) for r in rep["pass_c"] if r["variant"] == "per_column_pair"]
        assert shapes == [(1, 2, 1)]
        assert "groups_ca" not in rep
    monkeypatch.setenv("R2D3C_GROUPS", "0,1,0,0,2,4")  # a team wider than the two groups of a CTA, refused as ever
    with pytest.raises(gpu.R2D3CError):
        gpu.Context(params(1024, iflow=0)[1], gpu.FP32)


@pytest.mark.parametrize("n", [64, 256])
def test_shape_of_pass_c_with_pass_a(gpu, monkeypatch, n):
    rep = _report(gpu, n)
    assert rep["fused_ca"]
    timed = [r for r in rep["pass_c"] if "us_with_a" in r]
    # only shapes near the fastest without it are timed with it: creating a context pays for each
    pairs = [r for r in rep["pass_c"] if r["variant"] == "per_column_pair"]
    near = 1.15 * min(r["us"] for r in pairs)
    assert all(("us_with_a" in r) == (r["us"] <= near) for r in pairs if abs(r["us"] - near) > 0.02)
    assert len(timed) < len(pairs)
    best = min(timed, key=lambda r: r["us_with_a"])
    chosen = [r for r in timed
              if (r["groups"], r["chunks"], r["team"]) == (rep["groups_ca"], rep["chunks_ca"], rep["team_ca"])]
    assert chosen and chosen[0]["us_with_a"] == best["us_with_a"]
    monkeypatch.setenv("R2D3C_GROUPS", "0,1,0,2,2,2")
    rep = _report(gpu, n)
    assert (rep["groups_ca"], rep["chunks_ca"], rep["team_ca"]) == (2, 2, 2)
