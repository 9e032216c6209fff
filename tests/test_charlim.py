"""The characteristic limiter's shared-reciprocal division and its sparse
eigenvector products (csrc/gdf_charlim.cuh), compiled for the host and compared
value for value with the IEEE quotient and with the general path (eigen_left,
eigen_right, the full 8x8 products, minmod) over random and special states."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "freljord-cfd-arsenal_b200", "csrc")
dp = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(HERE, "native", "_build")
    os.makedirs(out, exist_ok=True)
    so, src = os.path.join(out, "libcharcheck.so"), os.path.join(HERE, "native", "charcheck.cpp")
    deps = [src] + [os.path.join(CSRC, f) for f in ("gdf_charlim.cuh", "gdf_physics.cuh")]
    if not os.path.exists(so) or os.path.getmtime(so) < max(map(os.path.getmtime, deps)):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-march=x86-64",
                        "-Wno-unknown-pragmas", "-o", so, src], check=True)
    return C.CDLL(so)


def P(a):
    return a.ctypes.data_as(dp)


def operands(kind, rng, n):
    if kind == "near_two":      # both significands just below 2: the quotient's first guess is furthest off
        return 2.0 - rng.integers(1, 4000, n) * 2.0 ** -52, 2.0 - rng.integers(1, 4000, n) * 2.0 ** -52
    if kind == "near_one":
        return 1.0 + rng.integers(0, 4000, n) * 2.0 ** -52, 1.0 + rng.integers(0, 4000, n) * 2.0 ** -52
    if kind == "wide":
        return (rng.uniform(1, 2, n) * 2.0 ** rng.integers(-1070, 1023, n) * rng.choice([-1, 1], n),
                rng.uniform(1, 2, n) * 2.0 ** rng.integers(-1022, 1023, n) * rng.choice([-1, 1], n))
    if kind == "special":
        v = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 2.0 ** -1022, 1.7e308, 1.0, -3.0, 0.4, 1e-300])
        a, b = np.meshgrid(v, v)
        return a.ravel().copy(), b.ravel().copy()
    a = rng.normal(0, 1, n) * 10.0 ** rng.uniform(-280, 280, n)   # b within the range, a almost anywhere in it
    return a, rng.uniform(1, 2, n) * 2.0 ** rng.integers(-60, 60, n) * rng.choice([-1, 1], n)


@pytest.mark.parametrize("kind", ["random", "near_two", "near_one", "wide", "special"])
def test_division_is_the_ieee_quotient(lib, kind):
    rng = np.random.default_rng(5)
    with np.errstate(all="ignore"):
        a, b = operands(kind, rng, 1_000_000)
        q = np.zeros_like(a)
        flagged = lib.cc_div(len(a), P(a), P(b), P(q))
        want = a / b
    assert np.all((q == want) | (np.isnan(q) & np.isnan(want)))
    if kind in ("near_two", "near_one"):
        assert flagged == 0
    elif kind == "random":
        assert flagged < 10   # (a within 1e-282 of zero)


def state(rng):
    rho = 10 ** rng.uniform(-2, 1)
    u, B = rng.uniform(-3, 3, 3), rng.uniform(-5, 5, 3) * rng.choice([1e-5, 0.1, 1, 6])
    for k in range(3):
        u[k] *= rng.random() > 0.25
        B[k] *= rng.random() > 0.25
    if rng.random() < 0.1:
        B[:] = 0.0
    p = 10 ** rng.uniform(-3, 3) * (-1 if rng.random() < 0.05 else 1)
    E = p / 0.4 + 0.5 * rho * (u @ u) + 0.5 * (B @ B)
    x = rng.normal(0, 1, (4, 8)) * 10 ** rng.uniform(-6, 1)
    x[:, rng.random(8) < 0.2] = 0.0
    if rng.random() < 0.05:
        x[rng.integers(4), rng.integers(8)] = rng.choice([np.inf, -np.inf, np.nan, 1e-200, 1e-308])
    if rng.random() < 0.03:
        rho = rng.choice([-rho, 0.0, np.nan, 1e200])
    return np.array([rho, *u, E, *B]), np.ascontiguousarray(x)


@pytest.mark.parametrize("ieee", [0, 1], ids=["shared", "ieee"])
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("variant", [(5 / 3, 0, 1, 0), (5 / 3, 1, 1, 0), (1.4, 0, 0, 0), (5 / 3, 0, 0, 1)],
                         ids=["p2", "p2_typo", "plain", "beta"])
def test_limited_slopes_equal_general_path(lib, direction, variant, ieee):
    gm, typo, ident, beta = variant
    rng = np.random.default_rng(11 + direction)
    ip = (C.c_int * 5)(direction, typo, ident, beta, ieee)
    took = refused = 0
    for _ in range(6000):
        prim, x = state(rng)
        prm = np.array([gm, 10 ** rng.uniform(-8, -1), 0.65])
        out = np.zeros(32)
        ok = lib.cc_limit(P(prm), ip, P(prim), P(x), P(out))
        if not ok:
            refused += 1
            continue
        took += 1
        fast, full = out[:16], out[16:]
        assert np.array_equal(fast, full), (prim, x, fast - full)
    # ordinary states are answered, the non-finite and out-of-range ones refused
    assert took > 5000 and refused > 30
