"""Which plain tile shapes the autotuner compares: all widths with trajectories enough to fill the rule's
sub-tiles on every SM, else that width alone (all widths would run the same claims, and noise would
choose the width of every later engine of the dimension)."""
import pytest

from tests.helpers import dimer_problem

pytestmark = pytest.mark.gpu


# the rule at d = 61: 32 columns, two CTAs on each of 148 SMs; d = 130: 16 (32 in one CTA per SM is a candidate
# too); d = 257: 16, one CTA per SM
@pytest.mark.parametrize("d,n,widths", [(61, 300, {32}), (61, 148 * 2 * 24 + 1, {8, 16, 32}), (130, 148 * 2 * 8, {16}),
                                        (130, 148 * 2 * 8 + 1, {8, 16, 32}), (257, 400, {16})])
def test_widths_compared(tmp_path, monkeypatch, d, n, widths):
    import os_d_b200 as q

    monkeypatch.setenv("QJX_TILE_CACHE", str(tmp_path / "tiles.txt"))
    P = dimer_problem(d - 1, g=1.0 / d, deep=2)
    best, table = q.autotune(P["U"], P["L"], [1.0], P["HE"], T=P["T"], n_traj=n, n_periods=1)
    assert {t["nc"] for t, _ in table} == widths
    assert min(table, key=lambda x: x[1])[0] == best and all(us > 0 for _, us in table)
    eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], None, P["T"], 40)  # takes the cached shape
    assert (tmp_path / "tiles.txt").read_text().startswith(f"0 {d} {best['nc']} {best['kb']} ")
    eng.close()
