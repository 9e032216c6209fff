"""The positivity limiter's own pass (one warp per listed cell, a lane per
GLL-mixed point) against the CPU oracle, value for value: states in which most
cells need the density part, the pressure part or both, on grids from one warp
to several rounds of the resident blocks, with the div-free reconstruction
fused into the pass and after it."""
import numpy as np
import pytest

import gdf
from oracle import Oracle

pytestmark = pytest.mark.gpu


def rough_state(cfg, seed, density):
    """Positive means (density, pressure) with modes large enough that many
    points lose pressure, and density too where asked."""
    rng = np.random.default_rng(seed)
    uh, bx, by = gdf._abi.new_state(cfg.nx, cfg.ny)
    sh = uh.shape[2:]
    uh[0, 0] = rng.uniform(0.5, 2.0, sh)
    uh[1:4, 0] = rng.normal(0, 1.0, (3,) + sh)
    uh[5:8, 0] = rng.normal(0, 1.0, (3,) + sh)
    p = 10.0 ** rng.uniform(-3, 1, sh)
    uh[4, 0] = (p / (cfg.gamma - 1) + 0.5 * (uh[1:4, 0] ** 2).sum(0) / uh[0, 0] + 0.5 * (uh[5:8, 0] ** 2).sum(0))
    size = 10.0 ** rng.uniform(-4, 0, sh)
    for n in range(8):
        for d in [1, 2, 3, 4, 5] + {5: [6, 8], 6: [7, 9]}.get(n, []):
            uh[n, d] = size * rng.normal(0, 0.6 if (n or density) else 0.05, sh)
    bx[:] = rng.normal(0, 0.3, bx.shape)
    by[:] = rng.normal(0, 0.3, by.shape)
    return uh, bx, by


@pytest.mark.parametrize("nx,ny", [(2, 2), (7, 5), (33, 18), (150, 131)])
@pytest.mark.parametrize("detector", [gdf.DETECT_ALL, gdf.DETECT_KXRCF], ids=["all", "kxrcf"])
@pytest.mark.parametrize("faceb", [0, 1])
@pytest.mark.parametrize("density", [False, True], ids=["pressure", "density"])
def test_limit_equals_oracle(nx, ny, detector, faceb, density):
    cfg, _ = gdf.problem_config(gdf.PROB_BLAST, nx, ny)
    cfg.detector, cfg.faceb_limiter = detector, faceb
    uh, bx, by = rough_state(cfg, 7 * nx + ny, density)
    o = Oracle(cfg)
    o.set_bc(uh)
    ou, ox, oy = uh.copy(), bx.copy(), by.copy()
    of = o.limit(ou, ox, oy)
    s = gdf.Solver(cfg)
    gu, gx, gy = uh.copy(), bx.copy(), by.copy()
    gf = s.limit(gu, gx, gy)
    # the limiter scaled a share of the cells (both parts are reached)
    assert (ou[4, 1] != uh[4, 1]).any()
    for a, b in ((gu, ou), (gx, ox), (gy, oy)):
        assert np.all((a == b) | (np.isnan(a) & np.isnan(b)))
    assert np.array_equal(gf, of)
    # the pass starts from an empty list each time
    gu2, gx2, gy2 = uh.copy(), bx.copy(), by.copy()
    s.set_trouble(np.zeros((ny, nx), np.int32))
    s.limit(gu2, gx2, gy2)
    assert np.array_equal(gu2, gu) and np.array_equal(gx2, gx) and np.array_equal(gy2, gy)
