"""Both forms of the residual (two lanes to a cell, one lane) on developed rotor
and blast states, either side of the line between them, against the oracle; and
a small grid's residual on caller-owned buffers, which is always the two-lane form."""
import numpy as np
import pytest

import gdf
from oracle import Oracle

pytestmark = pytest.mark.gpu


def equal(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("problem", [gdf.PROB_ROTOR, gdf.PROB_BLAST], ids=["rotor", "blast"])
@pytest.mark.parametrize("nx,ny", [(45, 37), (120, 118), (174, 160)])
def test_residual_and_step(problem, nx, ny):
    cfg, _ = gdf.problem_config(problem, nx, ny)
    s = gdf.Solver(cfg)
    s.upload(*Oracle(cfg).init_data(problem))
    s.prepare()
    s.advance(1e9, 12)
    uh, bx, by = s.download()
    trouble = s.trouble()
    o = Oracle(cfg)
    o.set_bc(uh)
    assert equal(s.lh(uh), o.lh(uh))
    o2, s2 = Oracle(cfg), gdf.Solver(cfg)
    s2.upload(uh, bx, by)
    s2.set_trouble(np.zeros_like(trouble))
    got = s2.step(1e9)
    ref = o2.step(uh, bx, by, 0.0, 1e9)
    assert got[:2] == ref[:2]
    for a, b in zip(s2.download(), (uh, bx, by)):
        assert equal(a, b)


# the largest grids of its scratch: square, and as long as it allows
@pytest.mark.parametrize("nx,ny", [(128, 128), (2, 5546), (5546, 2)])
def test_caller_owned_buffers(nx, ny):
    import torch
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
    rng = np.random.default_rng(nx)
    uh, _, _ = gdf._abi.new_state(nx, ny)
    uh[:, :6] = rng.normal(0, 0.05, uh[:, :6].shape)
    uh[0, 0] += 1.0
    uh[4, 0] += 3.0
    uh[5, 0] += 0.5
    d_uh = torch.from_numpy(uh).cuda()
    d_du = torch.empty_like(d_uh)
    gdf.lh_noalloc(cfg, d_uh.data_ptr(), d_du.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert equal(d_du.cpu().numpy(), Oracle(cfg).lh(uh))
