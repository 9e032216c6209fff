"""Copies through the pinned ring (csrc/gdf_stage.cu): states below, at and far
above the ring's chunk and size come back as they went, from pageable and from
pinned arrays, from several threads at once, and after the last handle (and
with it the ring) is gone."""
import threading

import numpy as np
import pytest

import gdf

pytestmark = pytest.mark.gpu


def state(nx, ny, seed):
    rng = np.random.default_rng(seed)
    uh, bx, by = gdf._abi.new_state(nx, ny)
    uh[:, :6] = rng.standard_normal(uh[:, :6].shape)
    uh[5, [6, 8]] = rng.standard_normal(uh[5, [6, 8]].shape)
    uh[6, [7, 9]] = rng.standard_normal(uh[6, [7, 9]].shape)
    bx[:], by[:] = rng.standard_normal(bx.shape), rng.standard_normal(by.shape)
    return uh, bx, by


def round_trip(nx, ny, seed, pinned=False):
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
    s = gdf.Solver(cfg)
    st = state(nx, ny, seed)
    if pinned:
        import torch
        st = tuple(torch.from_numpy(a).pin_memory().numpy() for a in st)
    for _ in range(2):
        s.upload(*st)
        back = s.download()
        for a, b in zip(st, back):
            assert np.array_equal(a, b)
        cells, bx, by = s.download_state()
        assert np.array_equal(cells[0], st[0][0, :6, 1:-1, 1:-1]) and np.array_equal(cells[5], st[0][7, :6, 1:-1, 1:-1])
        assert np.array_equal(bx, st[1]) and np.array_equal(by, st[2])
    s.close()


# six planes of (nx+2) x (ny+2) doubles per copy: 1 MB at 21845 cells, one chunk
# (4 MB) at 87381, the ring (16 MB) at 349525
@pytest.mark.parametrize("nx,ny", [(3, 2), (145, 146), (146, 146), (293, 293), (294, 294), (700, 531)])
@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
def test_round_trip(nx, ny, pinned):
    round_trip(nx, ny, nx, pinned)


def test_threads():
    errors = []

    def work(k):
        try:
            gdf.set_device(0)
            for r in range(3):
                round_trip(200 + 40 * k, 310 - 20 * k, 10 * k + r)
        except BaseException as e:   # reported by the main thread
            errors.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors


def test_dead_slot_is_found_whatever_its_place():
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, 300, 200)
    s = gdf.Solver(cfg)
    for n, d, j, i in [(0, 6, 0, 0), (4, 9, 201, 301), (5, 7, 100, 3), (6, 8, 7, 301), (7, 9, 201, 0)]:
        uh, bx, by = state(300, 200, 1)
        uh[n, d, j, i] = np.nan if n == 4 else 1e-300
        with pytest.raises(gdf.GdfError, match=f"mode {d + 1} of variable {n + 1}"):
            s.upload(uh, bx, by)
    uh, bx, by = state(300, 200, 1)
    uh[2, 7] = -0.0
    s.upload(uh, bx, by)
