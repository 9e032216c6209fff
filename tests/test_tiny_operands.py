"""States whose momenta and fields run from order one down through the
denormals (a disturbance spreading into a region at rest): the face solvers,
the residuals and the limiters take their shared-reciprocal path in some cells
and their IEEE path in others, and equal the oracle value for value in all."""
import numpy as np
import pytest

import gdf
from oracle import Oracle, OracleP3

pytestmark = pytest.mark.gpu


def fade(rng, sh):
    """Signed values with magnitudes from 1 to 1e-323, some exactly zero."""
    v = 10.0 ** rng.uniform(-323.5, 0, sh) * rng.choice([-1.0, 1.0], sh)
    v[rng.random(sh) < 0.1] = 0.0
    return v


def fill(uh, live, rng):
    sh = uh.shape[2:]
    for n in range(8):
        for d in range(uh.shape[1]):
            if live(n, d):
                uh[n, d] = fade(rng, sh) * (0.05 if d else 0.3)
    uh[0, 0] += 1.0
    uh[4, 0] += 3.0
    uh[5, 0] += 0.8


@pytest.mark.parametrize("flux", [gdf.FLUX_LF, gdf.FLUX_HLL, gdf.FLUX_HLLC, gdf.FLUX_HLLD])
@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 17), (66, 40)])
def test_p2(flux, nx, ny):
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
    cfg.flux_type, cfg.kxrcf_sticky = flux, 0
    uh, bx, by = gdf._abi.new_state(nx, ny)
    rng = np.random.default_rng(nx + flux)
    fill(uh, lambda n, d: d < 6 or (n == 5 and d in (6, 8)) or (n == 6 and d in (7, 9)), rng)
    o, s = Oracle(cfg), gdf.Solver(cfg)
    o.set_bc(uh)
    for a, b in ((s.lh(uh), o.lh(uh)), *zip(s.lhez(uh), o.lhez(uh))):
        assert np.all((a == b) | (np.isnan(a) & np.isnan(b)))
    for detector in (gdf.DETECT_ALL, gdf.DETECT_KXRCF):
        c = cfg.copy()
        c.detector = detector
        ou, ox, oy = uh.copy(), bx.copy(), by.copy()
        gu, gx, gy = uh.copy(), bx.copy(), by.copy()
        of = Oracle(c).limit(ou, ox, oy)
        gf = gdf.Solver(c).limit(gu, gx, gy)
        assert np.array_equal(gu, ou) and np.array_equal(gx, ox) and np.array_equal(gy, oy)
        assert np.array_equal(gf, of)


@pytest.mark.parametrize("flux", [gdf.FLUX_LF, gdf.FLUX_HLL, gdf.FLUX_HLLC, gdf.FLUX_HLLD])
@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 17), (66, 40)])
def test_p3(flux, nx, ny):
    from gdf import p3
    cfg, _ = p3.p3_problem_config(gdf.PROB_ROTOR, nx, ny)
    cfg.flux_type = flux
    uh, bx, by = p3.p3_new_state(nx, ny)
    live = p3.p3_live_mask()
    rng = np.random.default_rng(nx + flux)
    fill(uh, lambda n, d: live[n, d], rng)
    bx[:], by[:] = fade(rng, bx.shape), fade(rng, by.shape)
    o, s = OracleP3(cfg), p3.P3Solver(cfg)
    o.set_bc(uh, bx, by)
    for a, b in zip(s.lh(uh, bx, by), o.lh(uh, bx, by)):
        assert np.all((a == b) | (np.isnan(a) & np.isnan(b)))
    ou, ox, oy = uh.copy(), bx.copy(), by.copy()
    gu, gx, gy = uh.copy(), bx.copy(), by.copy()
    o.limit(ou, ox, oy)
    s.limit(gu, gx, gy)
    i = (slice(None), slice(None), slice(1, -1), slice(1, -1))
    assert np.array_equal(gu[i], ou[i])
