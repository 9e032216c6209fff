"""That the states of test_pp_pass reach both parts of the positivity limiter:
against the oracle with the limiter off, the density part changes modes of
density in some cells, and the pressure part scales the momenta and the energy
in some cells whose density it leaves alone."""
import numpy as np
import pytest

import gdf
from oracle import Oracle
from test_pp_pass import rough_state


@pytest.mark.parametrize("nx,ny", [(7, 5), (33, 18), (150, 131)])
@pytest.mark.parametrize("detector", [gdf.DETECT_ALL, gdf.DETECT_KXRCF], ids=["all", "kxrcf"])
@pytest.mark.parametrize("density", [False, True], ids=["pressure", "density"])
def test_both_parts(nx, ny, detector, density):
    out = []
    for pp in (1, 0):
        cfg, _ = gdf.problem_config(gdf.PROB_BLAST, nx, ny)
        cfg.detector, cfg.faceb_limiter, cfg.pp_limiter = detector, 1, pp
        uh, bx, by = rough_state(cfg, 7 * nx + ny, density)
        o = Oracle(cfg)
        o.set_bc(uh)
        o.limit(uh, bx, by)
        out.append(uh[:, 1:6, 1:-1, 1:-1])
    on, off = out
    rho = (on[0] != off[0]).any(0)
    rest = (on[1:5] != off[1:5]).any((0, 1))
    scaled = rest & ~rho
    assert rho.any() if density else scaled.any()
    # the pressure part acts on its own somewhere, on the density states too
    assert scaled.any() or nx * ny < 100
