"""KXRCF's bounds of the cell maximum at the ends of the number range: an energy
whose square overflows, and thresholds so far from one that the square of
threshold times length leaves the range. Flags equal the oracle's."""
import numpy as np
import pytest

import gdf
from oracle import Oracle

pytestmark = pytest.mark.gpu


# energies around 1e154, where squares pass 1e308; thresholds Ck over the
# jump ratios that occur (some 1 to 1000), scaled with the energy or not
@pytest.mark.parametrize("scale", [1.0, 1e150, 3e153, 1e154, 1e156, 1e300])
@pytest.mark.parametrize("ck", [1.0, 10.0, 100.0, 1e-160, 1e160])
def test_flags_equal_oracle(scale, ck):
    nx, ny = 33, 18
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
    cfg.kxrcf_ck, cfg.kxrcf_sticky, cfg.pp_limiter, cfg.faceb_limiter = ck, 0, 0, 0
    rng = np.random.default_rng(5)
    uh, bx, by = gdf._abi.new_state(nx, ny)
    sh = uh.shape[2:]
    uh[0, 0] = 1.0
    uh[1:3, 0] = rng.normal(0, 0.3, (2,) + sh)      # inflow through some faces
    uh[4, 0] = 2.0 + rng.normal(0, 0.3, sh)
    uh[4, 1:6] = rng.normal(0, 1.0, (5,) + sh)
    # only the energy jumps within a cell's reach of the threshold
    uh[4] *= scale
    o, s = Oracle(cfg), gdf.Solver(cfg)
    o.set_bc(uh)
    of = o.limit(uh.copy(), bx.copy(), by.copy())
    gf = s.limit(uh.copy(), bx.copy(), by.copy())
    gate = 7 << 24
    assert np.array_equal(gf & gate, of & gate)
    if scale == 1.0 and 1.0 <= ck <= 100.0:
        assert 0 < np.count_nonzero(of & gate) < of.size   # the thresholds lie among the ratios
