"""Residuals of states in which some values are infinite or so large that
fluxes overflow. The zeros of the basis decide there which entries of Lh turn
NaN (0 x inf): every form of a residual kernel leaves out the same zeros."""
import numpy as np
import pytest

import gdf
from oracle import OracleCy, OracleP3

pytestmark = pytest.mark.gpu


def spoil(uh, live, rng, how):
    """A smooth state of order one, then (how "inf", "huge") a few modes made so."""
    sh = uh.shape[2:]
    for n in range(8):
        for d in range(uh.shape[1]):
            if live(n, d):
                uh[n, d] = rng.normal(0, 0.05 if d else 0.3, sh)
    uh[0, 0] += 1.2
    uh[4, 0] += 3.0
    uh[5, 0] += 0.5
    if how == "none":
        return
    for n in range(8):
        for d in range(uh.shape[1]):
            if live(n, d):
                hit = rng.random(sh) < 0.003
                if how == "inf":
                    uh[n, d][hit] = rng.choice([np.inf, -np.inf], hit.sum())
                else:
                    uh[n, d][hit] *= 10.0 ** rng.uniform(150, 300, hit.sum())


def p2_live(n, d):
    return d < 6 or (n == 5 and d in (6, 8)) or (n == 6 and d in (7, 9))


# up to 28416 cells, ghosts included, two lanes take a cell, above it one lane:
# a block of a large grid and the small grid of the same cells and neighbours
@pytest.mark.parametrize("how", ["inf", "huge"])
@pytest.mark.parametrize("flux", [gdf.FLUX_LF, gdf.FLUX_HLL, gdf.FLUX_HLLC, gdf.FLUX_HLLD])
def test_p2_forms_agree(flux, how):
    def lh(uh):
        nx, ny = uh.shape[3] - 2, uh.shape[2] - 2
        cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
        cfg.flux_type = flux
        cfg.xa, cfg.xb, cfg.ya, cfg.yb = 0.0, nx / 128, 0.0, ny / 128   # the same cell size at any nx, ny
        return gdf.Solver(cfg).lh(uh)

    uh, _, _ = gdf._abi.new_state(200, 160)
    spoil(uh, p2_live, np.random.default_rng(flux), how)
    big = lh(uh)
    assert not np.isfinite(big).all()
    for nx, ny, i, j in ((40, 41, 0, 0), (150, 120, 31, 17), (7, 5, 190, 150)):
        small = lh(np.ascontiguousarray(uh[:, :, j:j + ny + 2, i:i + nx + 2]))
        inner = (slice(None), slice(None), slice(1, -1), slice(1, -1))
        assert np.array_equal(small[inner], big[:, :, j + 1:j + ny + 1, i + 1:i + nx + 1], equal_nan=True)


# the oracle multiplies by every zero
@pytest.mark.parametrize("how", ["inf", "huge"])
@pytest.mark.parametrize("flux", [gdf.FLUX_LF, gdf.FLUX_HLL, gdf.FLUX_HLLC, gdf.FLUX_HLLD])
@pytest.mark.parametrize("nx,ny", [(7, 5), (33, 18)])
def test_p3_equals_oracle(nx, ny, flux, how):
    from gdf import p3
    cfg, _ = p3.p3_problem_config(gdf.PROB_ROTOR, nx, ny)
    cfg.flux_type = flux
    uh, bx, by = p3.p3_new_state(nx, ny)
    live = p3.p3_live_mask()
    spoil(uh, lambda n, d: live[n, d], np.random.default_rng(nx + flux), how)
    for a, b in zip(p3.P3Solver(cfg).lh(uh, bx, by), OracleP3(cfg).lh(uh, bx, by)):
        assert np.array_equal(a, b, equal_nan=True)


# r B / r on the axis: a face there at an even nr
@pytest.mark.parametrize("nr,nz,lphi", [(2, 3, 1), (16, 9, 2), (34, 20, 1)])
@pytest.mark.parametrize("flux", [0, 1, 2], ids=["central", "lf", "hll"])
def test_cylindrical_axis_equals_oracle(flux, nr, nz, lphi):
    from gdf import cy
    cfg, _ = cy.cy_problem_config(cy.CY_SMOOTH_VORTEX, nr, nz, lphi)   # r from -5 to 5
    cfg.flux_type = flux
    assert nr % 2 or cfg.ra + (nr // 2) * ((cfg.rb - cfg.ra) / nr) == 0.0
    uh, br, bz = cy.cy_new_state(nr, nz, lphi)
    live = cy.cy_live_mask()
    spoil(uh, lambda n, d: live[n, d], np.random.default_rng(nr + flux), "none")
    got = cy.CySolver(cfg).lh(uh, br, bz)
    assert np.isinf(got[0]).any()
    for a, b in zip(got, OracleCy(cfg).lh(uh.copy(), 0.0)):
        assert np.array_equal(a, b, equal_nan=True)


# off the axis, with infinite and overflowing fluxes
@pytest.mark.parametrize("nr,nz,lphi", [(7, 5, 2), (16, 9, 4), (33, 18, 1)])
@pytest.mark.parametrize("how", ["inf", "huge"])
@pytest.mark.parametrize("flux", [0, 1, 2], ids=["central", "lf", "hll"])
def test_cylindrical_equals_oracle(flux, how, nr, nz, lphi):
    from gdf import cy
    cfg, _ = cy.cy_problem_config(cy.CY_SMOOTH_VORTEX, nr, nz, lphi)
    cfg.flux_type, cfg.ra, cfg.rb = flux, 1.0, 11.0
    uh, br, bz = cy.cy_new_state(nr, nz, lphi)
    live = cy.cy_live_mask()
    spoil(uh, lambda n, d: live[n, d], np.random.default_rng(nr + flux), how)
    for a, b in zip(cy.CySolver(cfg).lh(uh, br, bz), OracleCy(cfg).lh(uh.copy(), 0.0)):
        assert np.array_equal(a, b, equal_nan=True)
