"""Host copies of every kind of handle once the pinned ring exists (a
prediction on 69 MB makes all of its slots; a second handle keeps it), and of
the call that makes it: what is read back is what was written."""
import numpy as np
import pytest

import gdf

pytestmark = pytest.mark.gpu


@pytest.fixture
def ring():
    m = gdf.Mlp(0)
    X = np.random.default_rng(0).standard_normal((200000, gdf.NFEAT), dtype=np.float32)
    p = m.predict(X)                       # the call that makes the ring
    parts = np.concatenate([m.predict(X[k:k + 2500]) for k in range(0, len(X), 2500)])   # 0.9 MB each: plain copies
    assert np.array_equal(p, parts)
    assert np.array_equal(m.predict(X), p)
    yield m
    m.close()


def random_like(live, arrays, seed):
    rng = np.random.default_rng(seed)
    uh = arrays[0]
    for n in range(8):
        for d in range(uh.shape[1]):
            if live(n, d):
                uh[n, d] = rng.standard_normal(uh[n, d].shape)
    for a in arrays[1:]:
        a[:] = rng.standard_normal(a.shape)
    return arrays


def p2_live(n, d):
    return d < 6 or (n == 5 and d in (6, 8)) or (n == 6 and d in (7, 9))


def check(upload, download, state):
    for _ in range(2):
        upload(*state)
        for a, b in zip(download(), state):
            assert np.array_equal(a, b)


# a variable's run of planes from just over 1 MiB (one chunk) to beyond four
@pytest.mark.parametrize("nx,ny", [(146, 146), (293, 293), (294, 294), (700, 531)])
def test_p2_and_ensemble(ring, nx, ny):
    cfg, _ = gdf.problem_config(gdf.PROB_ROTOR, nx, ny)
    st = random_like(p2_live, gdf._abi.new_state(nx, ny), nx)
    s = gdf.Solver(cfg)
    check(s.upload, s.download, st)
    e = gdf.Ensemble([cfg, cfg])
    check(lambda *a: e.upload(1, *a), lambda: e.download(1), st)


@pytest.mark.parametrize("nx,ny", [(113, 113), (229, 227), (500, 333)])
def test_p3(ring, nx, ny):
    from gdf import p3
    live = p3.p3_live_mask()
    cfg, _ = p3.p3_problem_config(gdf.PROB_ROTOR, nx, ny)
    st = random_like(lambda n, d: live[n, d], p3.p3_new_state(nx, ny), nx)
    s = p3.P3Solver(cfg)
    check(s.upload, s.download, st)


@pytest.mark.parametrize("nr,nz,lphi", [(98, 98, 1), (227, 225, 1), (150, 100, 4)])
def test_cylindrical(ring, nr, nz, lphi):
    from gdf import cy
    live = cy.cy_live_mask()
    cfg, _ = cy.cy_problem_config(cy.CY_ORSZAG_TANG, nr, nz, lphi)
    st = random_like(lambda n, d: live[n, d], cy.cy_new_state(nr, nz, lphi), nr)
    s = cy.CySolver(cfg)
    check(s.upload, s.download, st)


def test_training_is_the_same_with_and_without(ring):
    rng = np.random.default_rng(3)
    X = rng.standard_normal((70000, gdf.NFEAT), dtype=np.float32)
    y = (X[:, 0] > 0).astype(np.float32)
    p0 = gdf.Mlp(5).params()

    def train():
        m = gdf.Mlp(1)
        m.set_params(p0)
        loss = m.train(X, y, epochs=2, batch=2048, lr=1e-3, seed=3)
        return loss, m.params()

    with_ring = train()
    ring.close()                           # the last holder: the copies of 25 MB are plain now
    without = train()
    assert np.array_equal(with_ring[0], without[0]) and np.array_equal(with_ring[1], without[1])
