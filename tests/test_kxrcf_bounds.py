"""KXRCF's decision by bounds of the cell maximum (csrc/gdf_device.cuh
kxrcf_flag) against the oracle's full evaluation: states whose jump ratios lie
below, above and between the bounds for thresholds Ck over twelve decades,
including the shipped Ck = 0 and exact zero jumps."""
import numpy as np
import pytest

import gdf
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 3), (33, 18), (65, 40)])
@pytest.mark.parametrize("ck", [0.0, 1e-6, 1.0, 30.0, 1e6])
def test_flags_equal_oracle(nx, ny, ck):
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
    cfg.kxrcf_ck, cfg.kxrcf_sticky, cfg.pp_limiter = ck, 0, 0
    rng = np.random.default_rng(3 * nx + ny)
    uh, bx, by = gdf._abi.new_state(nx, ny)
    sh = uh.shape[2:]
    smooth = 10.0 ** rng.uniform(-12, 0, sh)           # jump sizes from round-off to order one
    for n in range(8):
        uh[n, 0] = (2.0 if n in (0, 4) else 0.3) + smooth * rng.normal(0, 1, sh)
        for d in [1, 2, 3, 4, 5] + {5: [6, 8], 6: [7, 9]}.get(n, []):
            uh[n, d] = smooth * rng.normal(0, 0.3, sh)
    uh[4, 0] += 3.0
    uh[3] = uh[7] = 0.0                                 # no flow or field out of the plane
    uh[1:3, :, : ny // 2] = 0.0                         # a region at rest: no inflow face
    o = Oracle(cfg)
    o.set_bc(uh)
    ou, ox, oy = uh.copy(), bx.copy(), by.copy()
    of = o.limit(ou, ox, oy)
    gu, gx, gy = uh.copy(), bx.copy(), by.copy()
    gf = gdf.Solver(cfg).limit(gu, gx, gy)
    assert np.array_equal(gf, of)
    assert np.all((gu == ou) | (np.isnan(gu) & np.isnan(ou))) and np.array_equal(gx, ox) and np.array_equal(gy, oy)
