"""The pinned ring behind the library's host copies (csrc/gdf_stage.cu) built for
the host on a fake CUDA runtime (tests/native/fakecuda) whose copies run late
and whose events know their device: which ring a copy takes, when there is one,
and that it is given back."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "freljord-cfd-arsenal_b200", "csrc")


@pytest.fixture(scope="module")
def lib():
    native = os.path.join(HERE, "native")
    out = os.path.join(native, "_build")
    os.makedirs(out, exist_ok=True)
    so, src = os.path.join(out, "libstagecheck.so"), os.path.join(native, "stagecheck.cpp")
    deps = [src, os.path.join(native, "fakecuda", "cuda_runtime.h"), os.path.join(CSRC, "gdf_stage.cu"),
            os.path.join(CSRC, "gdf_stage.h")]
    if not os.path.exists(so) or os.path.getmtime(so) < max(map(os.path.getmtime, deps)):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(native, "fakecuda"),
                        "-o", so, src], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("check", ["other_device_current", "given_back", "plain", "failed_record", "when_made"])
def test_check(lib, check):
    assert getattr(lib, "check_" + check)() == 0
