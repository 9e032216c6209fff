"""The work a user has this framework do, as cases that can be timed and
compared: runs of the P2 solver (graph-replayed segments, a coupled host that
round-trips the state every step, one residual on caller-owned device
buffers), the reference's routines on host arrays, the ensemble, the k = 3 and
the cylindrical variant, and the learned indicator's training and inference.

Every run() starts from the inputs that prepare() made, so it can be repeated:
the state is uploaded (or projected on the device), advanced and downloaded, as
a program that restarts, couples or stores frames does.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "freljord-cfd-arsenal_b200"))
import gdf  # noqa: E402
from gdf import cy, p3  # noqa: E402
from gdf.indicator import Labeller, load_net  # noqa: E402

PROBLEM = {"ot": gdf.PROB_ORSZAG_TANG, "rotor": gdf.PROB_ROTOR, "blast": gdf.PROB_BLAST,
           "cloud": gdf.PROB_CLOUD_SHOCK}
FLUX = {"lf": gdf.FLUX_LF, "hll": gdf.FLUX_HLL, "hllc": gdf.FLUX_HLLC, "hlld": gdf.FLUX_HLLD}

# operations of one RK3 step per cell (+ - * / and square roots of the method,
# counted on the CPU restatement)
STEP_FLOPS = {"ot": 93.6e3, "rotor": 153.5e3, "blast": 156.2e3, "cloud": 93.6e3}


def listed():
    return [
        # one Lh on device buffers of the caller, the smallest call there is:
        # launches and the call's own host work count
        {"name": "residual_64_hll", "kind": "residual", "problem": "ot", "flux": "hll", "nx": 64, "ny": 64},
        # Orszag-Tang at the resolution the reference quotes, every cell limited
        {"name": "ot_128", "kind": "segment", "problem": "ot", "nx": 128, "ny": 128, "warm": 10, "steps": 40,
         "learned": False, "swirl": False},
        # the rotor once it has developed: HLLD, KXRCF + TVB, positivity limiter
        {"name": "rotor_512", "kind": "segment", "problem": "rotor", "nx": 512, "ny": 512, "warm": 100, "steps": 16,
         "learned": False, "swirl": False},
        # an odd grid with flow and field out of the plane (no exact zeros)
        {"name": "rotor_swirl_251x187", "kind": "segment", "problem": "rotor", "nx": 251, "ny": 187, "warm": 60,
         "steps": 30, "learned": False, "swirl": True},
        # the strong blast at full size with the learned gate, from its start
        {"name": "blast_2048_learned", "kind": "start", "problem": "blast", "nx": 2048, "ny": 2048, "steps": 8,
         "learned": True},
        # a host that exchanges the state with the solver at every step
        {"name": "blast_512_coupled", "kind": "coupled", "problem": "blast", "nx": 512, "ny": 512, "warm": 80,
         "steps": 6, "learned": True, "swirl": False},
        # eight problems of uneven size advanced together
        {"name": "ensemble_8", "kind": "ensemble", "instances": 8, "lo": 64, "hi": 160, "steps": 24},
        # the k = 3 variant on its cloud shock
        {"name": "p3_cloud_480x240", "kind": "p3", "problem": "cloud", "nx": 480, "ny": 240, "steps": 16},
        # the cylindrical variant in the reference's own configuration
        {"name": "cy_ot_192x2", "kind": "cy", "nr": 192, "nz": 192, "lphi": 1, "steps": 48},
        # the reference's routines one by one on host arrays (how the
        # indicator's training data is labelled)
        {"name": "routines_192", "kind": "routines", "problem": "blast", "nx": 192, "ny": 192},
        # training and inference of the indicator
        {"name": "mlp_train_65536", "kind": "mlp_train", "samples": 65536, "batch": 2048, "epochs": 2},
        {"name": "mlp_predict_200000", "kind": "mlp_predict", "samples": 200000},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["residual", "segment", "segment", "segment", "start", "coupled", "ensemble", "p3", "cy",
                       "routines", "mlp_train", "mlp_predict"])
    if kind == "residual":
        return {"kind": kind, "problem": rng.choice(["ot", "rotor", "blast"]), "flux": rng.choice(sorted(FLUX)),
                "nx": _log_int(rng, 8, 128), "ny": _log_int(rng, 8, 128)}
    if kind == "segment":
        problem = rng.choice(["ot", "rotor", "blast"])
        nx, ny = _log_int(rng, 32, 640), _log_int(rng, 32, 640)
        return {"kind": kind, "problem": problem, "nx": nx, "ny": ny, "warm": rng.choice([5, 20, 60]),
                "steps": max(4, min(40, 4_000_000 // (nx * ny))), "learned": problem == "blast" and rng.random() < 0.5,
                "swirl": rng.random() < 0.5}
    if kind == "start":
        nx, ny = _log_int(rng, 256, 1536), _log_int(rng, 256, 1536)
        return {"kind": kind, "problem": "blast", "nx": nx, "ny": ny, "steps": 8, "learned": rng.random() < 0.5}
    if kind == "coupled":
        return {"kind": kind, "problem": rng.choice(["rotor", "blast"]), "nx": _log_int(rng, 64, 640),
                "ny": _log_int(rng, 64, 640), "warm": 40, "steps": 4, "learned": False, "swirl": rng.random() < 0.5}
    if kind == "ensemble":
        lo = rng.randint(32, 96)
        return {"kind": kind, "instances": rng.randint(4, 16), "lo": lo, "hi": lo + rng.randint(16, 128), "steps": 16}
    if kind == "p3":
        return {"kind": kind, "problem": rng.choice(["ot", "rotor", "cloud"]), "nx": _log_int(rng, 48, 512),
                "ny": _log_int(rng, 48, 320), "steps": 10}
    if kind == "cy":
        lphi = rng.choice([1, 1, 2, 4])
        return {"kind": kind, "nr": _log_int(rng, 32, 256 // lphi), "nz": _log_int(rng, 32, 256 // lphi),
                "lphi": lphi, "steps": 24}
    if kind == "routines":
        return {"kind": kind, "problem": rng.choice(["rotor", "blast"]), "nx": _log_int(rng, 48, 256),
                "ny": _log_int(rng, 48, 256)}
    if kind == "mlp_train":
        return {"kind": kind, "samples": _log_int(rng, 4096, 131072), "batch": rng.choice([512, 1000, 2048, 4096]),
                "epochs": 1}
    return {"kind": kind, "samples": _log_int(rng, 1000, 400000)}


# ----------------------------------------------------------------- inputs --

def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _smooth(rng, ny, nx):
    """A smooth field in [-1, 1] on ny x nx cells: three seeded waves."""
    y, x = np.mgrid[0:ny, 0:nx]
    y, x = (y + 0.5) / ny, (x + 0.5) / nx
    f = np.zeros((ny, nx))
    for _ in range(3):
        kx, ky = rng.integers(1, 4, 2)
        f += np.sin(2 * np.pi * (kx * x + ky * y) + rng.uniform(0, 2 * np.pi)) / 3
    return f


def _blast_params(rng):
    """The benchmark blast moved and weakened or strengthened a little."""
    b = 100 / np.sqrt(8 * np.pi) * rng.uniform(0.8, 1.1)
    return np.array([rng.uniform(-0.05, 0.05), rng.uniform(-0.05, 0.05), 0.1, 1000.0 * rng.uniform(0.6, 1.2), 0.1,
                     1.0, b, b])


def _config(case):
    cfg, tend = gdf.problem_config(PROBLEM[case["problem"]], case["nx"], case["ny"])
    if case.get("learned"):
        cfg.detector = gdf.DETECT_LEARNED
    if "flux" in case:
        cfg.flux_type = FLUX[case["flux"]]
    return cfg, (tend if case["problem"] != "rotor" else 1e9)


def _solver(case, cfg):
    s = gdf.Solver(cfg)
    if case.get("learned"):
        net, lo, hi = load_net()
        s.set_indicator(net, lo, hi)
    return s


def _scale_momenta(u, rng, ny, nx):
    """The momenta of u (variable, mode, ..., ny, nx) scaled by 1 + 2% of a
    smooth field, the mean energies with them: the pressure stays."""
    f = 1.0 + 0.02 * _smooth(rng, ny, nx)
    u[4, 0] += 0.5 * (u[1, 0] ** 2 + u[2, 0] ** 2 + u[3, 0] ** 2) / u[0, 0] * (f * f - 1.0)
    u[1:4] *= f


def _perturb(cells, rng, swirl):
    """Seeded inputs of the same kind: the momenta scaled; with swirl, a
    smooth flow and field out of the plane (their energy added)."""
    ny, nx = cells.shape[2:]
    _scale_momenta(cells, rng, ny, nx)
    if swirl:
        w, bz = 0.2 * _smooth(rng, ny, nx), 0.2 * _smooth(rng, ny, nx)
        cells[3, :6] += cells[0, :6] * w
        cells[5, 0] += bz
        cells[4, 0] += 0.5 * cells[0, 0] * w * w + 0.5 * bz * bz


def _developed(case, seed):
    """A handle and its compact state after `warm` steps, perturbed."""
    rng = np.random.default_rng(seed)
    cfg, tend = _config(case)
    s = _solver(case, cfg)
    s.init_device(PROBLEM[case["problem"]], _blast_params(rng) if case["problem"] == "blast" else None)
    s.prepare()
    s.advance(tend, case["warm"])
    cells, bx, by = s.download_state()
    _perturb(cells, rng, case.get("swirl"))
    hold = tuple(_pinned(a) for a in (cells, bx, by))
    out = tuple(_pinned(np.zeros_like(a)) for a in (cells, bx, by))
    return {"s": s, "tend": tend, "in": hold, "out": out, "t": s.t, "trouble": s.trouble()}


def _host_state(case, seed):
    """Reference arrays (uh, bx, by) after a few steps of the problem, the
    momenta scaled as in _perturb, the ghost cells set as set_bc does."""
    rng = np.random.default_rng(seed)
    natural = {k: v for k, v in case.items() if k != "flux"}
    cfg, tend = _config(natural)
    s = _solver(natural, cfg)
    s.init_device(PROBLEM[case["problem"]], _blast_params(rng) if case["problem"] == "blast" else None)
    s.prepare()
    s.advance(tend, 20)
    uh, bx, by = s.download()
    s.close()
    _scale_momenta(uh[:, :, 1:-1, 1:-1], rng, case["ny"], case["nx"])
    lo, hi = (-2, 1) if cfg.bc_l == gdf.BC_PERIODIC else (1, -2)
    uh[..., 0], uh[..., -1] = uh[..., lo], uh[..., hi]
    uh[:, :, 0], uh[:, :, -1] = uh[:, :, lo], uh[:, :, hi]
    return _config(case)[0], tend, uh, bx, by


def _features(case, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((case["samples"], gdf.NFEAT), dtype=np.float32)
    y = (X[:, :8].sum(1) > 1.0).astype(np.float32)
    a1, a2, a3 = np.sqrt(6 / 154), np.sqrt(6 / 128), np.sqrt(6 / 65)
    p = np.concatenate([rng.uniform(-a1, a1, 90 * 64), np.zeros(64), rng.uniform(-a2, a2, 64 * 64), np.zeros(64),
                        rng.uniform(-a3, a3, 64), np.zeros(1)]).astype(np.float32)
    return X, y, p


def prepare(case, seed):
    kind = case["kind"]
    if kind == "residual":
        cfg, _, uh, _, _ = _host_state(case, seed)
        d_uh = torch.from_numpy(uh).cuda()
        return {"kind": kind, "cfg": cfg, "uh": d_uh, "du": torch.empty_like(d_uh)}
    if kind in ("segment", "coupled"):
        return dict(_developed(case, seed), kind=kind, steps=case["steps"])
    if kind == "start":
        cfg, tend = _config(case)
        s = _solver(case, cfg)
        out = tuple(torch.zeros(sh, dtype=torch.float64, pin_memory=True).numpy()
                    for sh in (s.state_shape(), (3, cfg.ny, cfg.nx + 1), (3, cfg.ny + 1, cfg.nx)))
        return {"kind": kind, "s": s, "tend": tend, "out": out, "steps": case["steps"],
                "problem": PROBLEM[case["problem"]], "params": _blast_params(np.random.default_rng(seed))}
    if kind == "ensemble":
        n = case["instances"]
        cfgs, states, ends = [], [], []
        for i in range(n):
            side = case["lo"] + (case["hi"] - case["lo"]) * i // max(1, n - 1)
            problem = ("ot", "rotor", "blast")[i % 3]
            cfg, tend = gdf.problem_config(PROBLEM[problem], side, side)
            cfg.flux_type, cfg.faceb_limiter, cfg.detector, cfg.kxrcf_ck = gdf.FLUX_HLLD, 1, gdf.DETECT_LEARNED, 1.0
            rng = np.random.default_rng([seed, i])
            uh, bx, by = gdf.init_data(cfg, PROBLEM[problem], _blast_params(rng) if problem == "blast" else None)
            _scale_momenta(uh[:, :6, 1:-1, 1:-1], rng, side, side)
            cfgs.append(cfg)
            states.append((uh, bx, by))
            ends.append(tend)
        e = gdf.Ensemble(cfgs)
        net, lo, hi = load_net()
        e.set_indicator(net, lo, hi)
        return {"kind": kind, "e": e, "states": states, "ends": ends, "steps": case["steps"]}
    if kind == "p3":
        rng = np.random.default_rng(seed)
        cfg, tend = p3.p3_problem_config(PROBLEM[case["problem"]], case["nx"], case["ny"])
        uh, bx, by = p3.p3_init_data(cfg, PROBLEM[case["problem"]])
        _scale_momenta(uh[..., 1:-1, 1:-1], rng, case["ny"], case["nx"])
        return {"kind": kind, "s": p3.P3Solver(cfg), "tend": tend, "in": (uh, bx, by), "steps": case["steps"]}
    if kind == "cy":
        rng = np.random.default_rng(seed)
        cfg, tend = cy.cy_problem_config(cy.CY_ORSZAG_TANG, case["nr"], case["nz"], case["lphi"])
        uh, br, bz = cy.cy_init_data(cfg, cy.CY_ORSZAG_TANG)
        _scale_momenta(uh[..., 1:-1, 1:-1], rng, case["nz"], case["nr"])
        return {"kind": kind, "s": cy.CySolver(cfg), "tend": tend, "in": (uh, br, bz), "steps": case["steps"]}
    if kind == "routines":
        cfg, _, uh, bx, by = _host_state(case, seed)
        return {"kind": kind, "lab": Labeller(cfg), "in": (uh, bx, by)}
    X, y, p = _features(case, seed)
    m = gdf.Mlp(0)
    m.set_params(p)
    return dict(case, m=m, X=X, y=y, p=p)


# -------------------------------------------------------------------- run --

def run(st):
    kind = st["kind"]
    if kind == "residual":
        gdf.lh_noalloc(st["cfg"], st["uh"].data_ptr(), st["du"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return st["du"]
    if kind == "segment":
        s = st["s"]
        s.upload_state(*st["in"])
        s.set_trouble(st["trouble"])
        s.set_time(st["t"])
        t, _ = s.advance(st["tend"], st["steps"])
        cells, bx, by = s.download_state(*st["out"])
        umax, div, pmin, gated = s.diagnostics()
        return {"cells": cells, "bx": bx, "by": by, "t": t, "umax": umax, "pmin": pmin, "gated": gated,
                "trouble": s.trouble()}
    if kind == "start":
        s = st["s"]
        s.init_device(st["problem"], st["params"])
        s.prepare()
        t, _ = s.advance(st["tend"], st["steps"])
        cells, bx, by = s.download_state(*st["out"])
        return {"cells": cells, "bx": bx, "by": by, "t": t}
    if kind == "coupled":
        s = st["s"]
        s.set_trouble(st["trouble"])
        s.set_time(st["t"])
        state, out = st["in"], st["out"]
        for _ in range(st["steps"]):
            s.upload_state(*state)
            t, dt, flags = s.step(st["tend"])
            s.download_state(*out)
            state = out
        return {"cells": out[0], "bx": out[1], "by": out[2], "t": t, "dt": dt, "flags": flags}
    if kind == "ensemble":
        e = st["e"]
        for i, u in enumerate(st["states"]):
            e.upload(i, *u)
        e.prepare()
        for i, tend in enumerate(st["ends"]):
            e.set_time(i, 0.0, tend)
        updates, running, _ = e.advance(st["steps"])
        return {"updates": updates, "running": running, "states": [e.download(i) for i in range(e.n)]}
    if kind in ("p3", "cy"):
        s = st["s"]
        s.upload(*st["in"])
        s.set_time(0.0)
        s.prepare()
        t, _ = s.advance(st["tend"], st["steps"])
        return {"t": t, "state": s.download()}
    if kind == "routines":
        X, y, kx, change = st["lab"].sample(*st["in"])
        return {"X": X, "y": y, "kxrcf": kx, "change": change}
    m = st["m"]
    m.set_params(st["p"])
    if kind == "mlp_train":
        losses = m.train(st["X"], st["y"], epochs=st["epochs"], batch=st["batch"], lr=1e-3, pos_weight=2.0, seed=3)
        return {"losses": losses, "params": m.params()}
    return m.predict(st["X"])


# ------------------------------------------------------- what it cannot skip

def work(case):
    """The arrays that go in and come out, and the method's operations."""
    kind = case["kind"]
    if kind == "residual":
        n = (case["nx"] + 2) * (case["ny"] + 2)
        return {"bytes": 2 * 52 * 8.0 * n, "flops": 0.25 * STEP_FLOPS[case["problem"]] * case["nx"] * case["ny"]}
    if kind in ("segment", "start", "coupled"):
        n, k = case["nx"] * case["ny"], case["steps"]
        moves = {"segment": 2, "start": 1, "coupled": 2 * k}[kind]
        return {"bytes": moves * 42 * 8.0 * n, "flops": STEP_FLOPS[case["problem"]] * n * k}
    if kind == "ensemble":
        m = case["instances"]
        sides = [case["lo"] + (case["hi"] - case["lo"]) * i // max(1, m - 1) for i in range(m)]
        n = float(sum(s * s for s in sides))
        return {"bytes": 2 * 86 * 8 * n, "flops": 150e3 * n * case["steps"]}
    if kind == "p3":
        n, k = case["nx"] * case["ny"], case["steps"]
        return {"bytes": 2 * 128 * 8.0 * n, "flops": 600e3 * n * k}
    if kind == "cy":
        n, k = 2 * case["lphi"] * case["nr"] * case["nz"], case["steps"]
        return {"bytes": 2 * 86 * 8.0 * n, "flops": 100e3 * n * k}
    if kind == "routines":
        n = (case["nx"] + 2) * (case["ny"] + 2)
        return {"bytes": (86 * 8 + 90 * 4) * 1.0 * n, "flops": 60e3 * n}
    per = 2.0 * (90 * 64 + 64 * 64 + 64) * case["samples"]
    if kind == "mlp_train":
        return {"bytes": 364.0 * case["samples"], "flops": 3 * per * case["epochs"]}
    return {"bytes": 364.0 * case["samples"], "flops": per}


# ------------------------------------------------------- 64-bit references --

def _basis(x, y):
    """The ten modal basis functions at (x, y) of the reference cell."""
    p2 = lambda v: v * v - 1 / 3  # noqa: E731
    p3_ = lambda v: v ** 3 - 0.6 * v  # noqa: E731
    one = np.ones_like(x * y)
    return np.stack([one, x * one, y * one, p2(x) * one, x * y, p2(y) * one, p3_(x) * one, p2(x) * y, x * p2(y),
                     p3_(y) * one])


def _basis_d(x, y):
    """Their derivatives in x and y."""
    z, one = np.zeros_like(x * y), np.ones_like(x * y)
    dx = [z, one, z, 2 * x * one, y * one, z, (3 * x * x - 0.6) * one, 2 * x * y, (y * y - 1 / 3) * one, z]
    dy = [z, z, one, z, x * one, 2 * y * one, z, (x * x - 1 / 3) * one, 2 * x * y, (3 * y * y - 0.6) * one]
    return np.stack(dx), np.stack(dy)


def _prim(q, gamma):
    u, v, w = q[1] / q[0], q[2] / q[0], q[3] / q[0]
    bb = q[5] ** 2 + q[6] ** 2 + q[7] ** 2
    return u, v, w, bb, (gamma - 1) * (q[4] - 0.5 * q[0] * (u * u + v * v + w * w) - 0.5 * bb)


def _flux(q, axis, gamma, minus_w=False):
    """Ideal-MHD flux; minus_w: the method's pressure on the upper side of a
    y face, which adds the w part of the kinetic energy."""
    u, v, w, bb, p = _prim(q, gamma)
    if minus_w:
        p = p + (gamma - 1) * q[0] * w * w
    un, bn = (u, q[5]) if axis == 0 else (v, q[6])
    pt = p + 0.5 * bb
    kb = u * q[5] + v * q[6] + w * q[7]
    f = [q[0] * un, q[1] * un - q[5] * bn, q[2] * un - q[6] * bn, q[3] * un - q[7] * bn, (q[4] + pt) * un - kb * bn,
         q[5] * un - u * bn, q[6] * un - v * bn, q[7] * un - w * bn]
    f[1 + axis] = f[1 + axis] + pt
    f[5 + axis] = np.zeros_like(un)
    return np.stack(f)


def _speeds(q, axis, gamma):
    u, v, w, bb, p = _prim(q, gamma)
    un, bn = (u, q[5]) if axis == 0 else (v, q[6])
    c2, b2 = np.abs(gamma * p / q[0]), bb / q[0]
    cf = np.sqrt(np.abs(0.5 * (c2 + b2 + np.sqrt((c2 + b2) ** 2 - 4 * c2 * bn ** 2 / q[0]))))
    return un + cf, un - cf


def _riemann(lo, hi, axis, cfg):
    f_lo, f_hi = _flux(lo, axis, cfg.gamma), _flux(hi, axis, cfg.gamma, minus_w=axis == 1)
    (a1, a2), (b1, b2) = _speeds(lo, axis, cfg.gamma), _speeds(hi, axis, cfg.gamma)
    sr, sl = np.maximum(a1, b1), np.minimum(a2, b2)
    if cfg.flux_type == gdf.FLUX_LF:
        return 0.5 * (f_lo + f_hi - np.maximum(np.abs(sr), np.abs(sl)) * (hi - lo))
    mid = (sr * f_lo - sl * f_hi + sl * sr * (hi - lo)) / (sr - sl)
    return np.where(sr < 0, f_hi, np.where(sl > 0, f_lo, mid))


def _residual(cfg, uh):
    """du of the semi-discrete P2 scheme (volume and surface integrals over
    the inverse mass matrix), LF or HLL fluxes."""
    x, wt = np.polynomial.legendre.leggauss(5)
    hx, hy = (cfg.xb - cfg.xa) / cfg.nx, (cfg.yb - cfg.ya) / cfg.ny
    gx, gy = np.meshgrid(x, x, indexing="ij")
    ph, (dx, dy) = _basis(gx, gy), _basis_d(gx, gy)
    inner = uh[:, :, 1:-1, 1:-1]
    du = np.zeros((8, 10) + inner.shape[2:])
    for a in range(5):
        for b in range(5):
            q = np.einsum("ndji,d->nji", inner, ph[:, a, b])
            fx, fy = _flux(q, 0, cfg.gamma), _flux(q, 1, cfg.gamma)
            c = 0.25 * wt[a] * wt[b]
            for d in range(10):
                du[:, d] += c * (fx * (dx[d, a, b] * 2 / hx) + fy * (dy[d, a, b] * 2 / hy))
    for g in range(5):
        r, l = _basis(np.float64(1), x[g]), _basis(np.float64(-1), x[g])
        u, d_ = _basis(x[g], np.float64(1)), _basis(x[g], np.float64(-1))
        rows, cols = uh[:, :, 1:-1, :], uh[:, :, :, 1:-1]
        f = _riemann(np.einsum("ndji,d->nji", rows[..., :-1], r), np.einsum("ndji,d->nji", rows[..., 1:], l), 0, cfg)
        h = _riemann(np.einsum("ndji,d->nji", cols[:, :, :-1], u), np.einsum("ndji,d->nji", cols[:, :, 1:], d_), 1, cfg)
        for d in range(10):
            du[:, d] -= 0.5 / hx * wt[g] * (f[..., 1:] * r[d] - f[..., :-1] * l[d])
            du[:, d] -= 0.5 / hy * wt[g] * (h[:, 1:] * u[d] - h[:, :-1] * d_[d])
    mm = np.array([1, 1 / 3, 1 / 3, 4 / 45, 1 / 9, 4 / 45, 4 / 175, 4 / 135, 4 / 135, 4 / 175])
    live = np.zeros((8, 10))
    live[:, :6] = 1
    live[5, [6, 8]] = live[6, [7, 9]] = 1
    out = np.zeros_like(uh)
    out[:, :, 1:-1, 1:-1] = du * (live / mm)[:, :, None, None]
    return out


def exact(case, seed):
    """The residual (LF, HLL) and the network's probabilities in plain numpy.
    Whole steps with the limiters, the HLLC/HLLD solvers, the other variants
    and training runs have none: many steps of thousands of operations per
    cell with branches take numpy longer than the comparison allows."""
    if case["kind"] == "residual" and case["flux"] in ("lf", "hll"):
        cfg, _, uh, _, _ = _host_state(case, seed)
        return _residual(cfg, uh)
    if case["kind"] == "mlp_predict":
        from math import sqrt
        X, _, p = _features(case, seed)
        X, p = torch.from_numpy(X).double(), torch.from_numpy(p).double()
        gelu = lambda z: 0.5 * z * (1 + torch.erf(z / sqrt(2)))  # noqa: E731
        w1, b1, w2, b2, w3, b3 = torch.split(p, [90 * 64, 64, 64 * 64, 64, 64, 1])
        h = gelu(gelu(X @ w1.reshape(90, 64) + b1) @ w2.reshape(64, 64) + b2)
        return torch.sigmoid(h @ w3 + b3)
    return None
