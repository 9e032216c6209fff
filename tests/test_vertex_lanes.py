"""The vertex solver with four lanes to a vertex (csrc/gdf_vertex.cuh), compiled
for the host, value for value against the one-thread solver: subsonic and
supersonic corners in both directions, no field, nearly equal states, tiny ones."""
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
    so, src = os.path.join(out, "libvertexcheck.so"), os.path.join(HERE, "native", "vertexcheck.cpp")
    deps = [src] + [os.path.join(CSRC, f) for f in ("gdf_vertex.cuh", "gdf_physics.cuh")]
    if not os.path.exists(so) or os.path.getmtime(so) < max(map(os.path.getmtime, deps)):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-march=x86-64",
                        "-Wno-unknown-pragmas", "-o", so, src], check=True)
    return C.CDLL(so)


def corners(kind, rng, n):
    m = 0.01 if kind == "near" else 1.0
    base = rng.uniform(0.5, 1.5, (n, 1, 1)) if kind == "near" else 1.0
    rho = base + m * rng.uniform(0.1 if m == 1 else 0, 2, (n, 4, 1))
    u = m * rng.standard_normal((n, 4, 3))
    if kind == "fast":
        u = u + rng.choice([-9.0, 0.0, 9.0], (n, 1, 3))
    B = m * rng.standard_normal((n, 4, 3))
    if kind == "no_field":
        B = np.zeros((n, 4, 3))
    if kind == "plane":             # no normal field in x, nothing out of the plane
        B[:, :, 0] = 0
        B[:, :, 2] = u[:, :, 2] = 0
    p = base + m * rng.uniform(0.05 if m == 1 else 0, 2, (n, 4, 1))
    if kind == "tiny":              # leaves rdiv's ranges
        rho, B = rho * 2.0 ** -70, B * 2.0 ** -500
    E = p / (5 / 3 - 1) + 0.5 * rho * (u ** 2).sum(2, keepdims=True) + 0.5 * (B ** 2).sum(2, keepdims=True)
    return np.ascontiguousarray(np.concatenate([rho, rho * u, E, B], axis=2))


@pytest.mark.parametrize("flux", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["plain", "fast", "near", "no_field", "plane", "tiny", "still"])
def test_four_lanes_equal_one_thread(lib, kind, flux):
    rng = np.random.default_rng(7)
    n = 4000
    U = corners("near" if kind == "still" else kind, rng, n)
    if kind == "still":             # four equal corners
        U = np.ascontiguousarray(np.repeat(U[:, :1], 4, axis=1))
    got, want, how = np.zeros(n), np.ones(n), np.zeros(n, np.int32)
    a = [x.ctypes.data_as(C.c_void_p) for x in (U, got, want, how)]
    lib.vertex_four(C.c_double(5 / 3), C.c_double(5 / 3), C.c_double(1e-6), flux, C.c_longlong(n), *a)
    assert np.array_equal(got, want, equal_nan=True)
    if kind in ("plain", "fast", "near"):
        assert how.mean() > 0.9     # the shared reciprocals take ordinary vertices
    if kind == "tiny":
        assert not how.any()        # the density is below rdiv's range
