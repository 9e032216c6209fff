"""The residual with two lanes to a cell (small grids) and with one, either side
of the line between them and at grids that end inside a half warp: the residual
and whole steps equal the oracle's value for value."""
import numpy as np
import pytest

import gdf
from oracle import Oracle

pytestmark = pytest.mark.gpu


def equal(a, b):
    return bool(np.all((a == b) | (np.isnan(a) & np.isnan(b))))


@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 5), (13, 2), (46, 31), (174, 158), (174, 160)])
def test_residual_and_step(nx, ny):
    cfg, _ = gdf.problem_config(gdf.PROB_ORSZAG_TANG, nx, ny)
    o, s = Oracle(cfg), gdf.Solver(cfg)
    uh, bx, by = o.init_data(gdf.PROB_ORSZAG_TANG)
    rng = np.random.default_rng(nx)
    live = np.zeros((8, uh.shape[1], 1, 1), bool)
    live[:, :6] = True
    for n, d in ((5, 6), (5, 8), (6, 7), (6, 9)):
        live[n, d] = True
    uh = uh + 1e-3 * live * rng.standard_normal(uh.shape)
    o.set_bc(uh)
    assert equal(s.lh(uh), o.lh(uh))
    s.upload(uh, bx, by)
    assert s.step(1e9)[:2] == o.step(uh, bx, by, 0.0, 1e9)[:2]
    for a, b in zip(s.download(), (uh, bx, by)):
        assert equal(a, b)
