"""The states of test_tiny_operands (momenta and fields from order one down
through the denormals) through the kernels it leaves out: the cylindrical
residual and limiter against the oracle, and the ensemble's step, whose residual
and limiter passes are its own, against the single-problem handle."""
import numpy as np
import pytest

import gdf
from oracle import OracleCy
from test_tiny_operands import fade, fill

pytestmark = pytest.mark.gpu


# lphi 1 and 4: prim_c, the projection of r B, the limiter and its refused
# cells, the divergence-free rebuild
@pytest.mark.parametrize("flux", [0, 1, 2], ids=["central", "lf", "hll"])
@pytest.mark.parametrize("nr,nz,lphi", [(2, 2, 1), (31, 17, 1), (20, 33, 4)])
def test_cylindrical(flux, nr, nz, lphi):
    from gdf import cy
    cfg, _ = cy.cy_problem_config(cy.CY_ORSZAG_TANG, nr, nz, lphi)
    cfg.flux_type = flux
    uh, br, bz = cy.cy_new_state(nr, nz, lphi)
    live = cy.cy_live_mask()
    rng = np.random.default_rng(nr + flux)
    fill(uh, lambda n, d: live[n, d], rng)
    br[:], bz[:] = fade(rng, br.shape), fade(rng, bz.shape)
    s = cy.CySolver(cfg)
    for a, b in zip(s.lh(uh, br, bz), OracleCy(cfg).lh(uh.copy(), 0.0)):
        assert np.array_equal(a, b, equal_nan=True)
    gu, gr, gz = uh.copy(), br.copy(), bz.copy()
    ou, orr, oz = uh.copy(), br.copy(), bz.copy()
    s.limit(gu, gr, gz)
    OracleCy(cfg).limit(ou, orr, oz)
    i = (slice(None),) * 3 + (slice(1, -1), slice(1, -1))
    assert np.array_equal(gu[i], ou[i]) and np.array_equal(gr, orr) and np.array_equal(gz, oz)


@pytest.mark.parametrize("mode", [0, 1], ids=["persistent", "per-phase"])
@pytest.mark.parametrize("detector", [gdf.DETECT_ALL, gdf.DETECT_KXRCF], ids=["all", "kxrcf"])
def test_ensemble(mode, detector):
    rng = np.random.default_rng(7 + detector)
    cfgs, states = [], []
    for k, (nx, ny) in enumerate([(2, 2), (31, 17), (66, 40), (40, 41)]):
        cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
        cfg.flux_type, cfg.detector = 1 + k, detector
        uh, bx, by = gdf._abi.new_state(nx, ny)
        fill(uh, lambda n, d: d < 6 or (n == 5 and d in (6, 8)) or (n == 6 and d in (7, 9)), rng)
        bx[:], by[:] = fade(rng, bx.shape), fade(rng, by.shape)
        cfgs.append(cfg)
        states.append((uh, bx, by))
    e = gdf.Ensemble(cfgs)
    e.set_mode(mode)
    for i, st in enumerate(states):
        e.upload(i, *st)
    e.prepare()
    for i in range(len(cfgs)):
        e.set_time(i, 0.0, 1e9)
    e.advance(2)
    for i, st in enumerate(states):
        s = gdf.Solver(cfgs[i])
        s.upload(*st)
        s.prepare()
        s.advance(1e9, 2)
        for a, b in zip(e.download(i), s.download()):
            assert np.array_equal(a, b)
