"""Rows per warp of the double-precision predictor: eif_tiles reports the rows that run, and all
of them (1 to 16, with partial last strips and walks) give the same bits."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, Simulation, cases

pytestmark = pytest.mark.gpu


def run(monkeypatch, grid, tiles=None, tune=None):
    for name, v in (("EIF_TILES", tiles), ("EIF_TUNE", tune)):
        if v is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, v)
    case = cases.poiseuille(itot=grid[0], jtot=grid[1], n=2, a=0.06, b=0.04, seed=3)
    with Simulation.from_case(case, precision=PREC_FP64) as s:
        s.advance(3)
        return [np.array(a) for a in s.pull_fluid()[:3]] + [np.array(s.pull_particles())], s.tiles()


# strips of 31 columns x rows at 8 warps on each of 152 SMs: one row per warp on the two small
# grids, two at 256 x 512, eight at 512 x 1024
@pytest.mark.parametrize("grid,default", [((64, 128), 1), ((54, 100), 1), ((96, 190), 1), ((256, 512), 2), ((512, 1024), 8)])
def test_rows_reported_and_results_equal(grid, default, gpu_lib, monkeypatch):
    want, t = run(monkeypatch, grid, tune="0")
    assert t["predictor_rows"] == default
    out, t = run(monkeypatch, grid)
    assert t["predictor_rows"] in (1, 2, 4, 8, 16)
    outs = [out]
    for rows in (4, 8, 16):
        out, t = run(monkeypatch, grid, tiles="%d,8,128" % rows)
        assert t["predictor_rows"] == rows
        outs.append(out)
    for out in outs:
        for a, b in zip(out, want):
            assert np.array_equal(a, b)
