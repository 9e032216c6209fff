"""Block shapes that kernels of different files rely on are checked when the
library is compiled: with one of the constants changed alone, the compiler
refuses the file that needs the other."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = "freljord-cfd-arsenal_b200"
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("source,old,new,file", [
    # the persistent stage kernel's shared memory: its own block, cell_item's stride
    ("gdf_device.cuh", "constexpr int CELL_BS = 64;", "constexpr int CELL_BS = 32;", "gdf_ensemble.cu"),
    ("gdf_ensemble.cu", "constexpr int ENS_BS = 64;", "constexpr int ENS_BS = 128;", "gdf_ensemble.cu"),
    # a tile's lanes against the two-lane residual's block
    ("gdf_device.cuh", "constexpr int PAIR_BS = 128,", "constexpr int PAIR_BS = 256,", "gdf_ensemble.cu")])
def test_refused(tmp_path, source, old, new, file):
    csrc = tmp_path / PKG / "csrc"
    shutil.copytree(os.path.join(REPO, PKG, "csrc"), csrc)
    shutil.copytree(os.path.join(REPO, "include"), tmp_path / "include")
    text = (csrc / source).read_text()
    assert text.count(old) == 1
    (csrc / source).write_text(text.replace(old, new))
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-ptx", "-o", os.devnull,
                        str(csrc / file)], capture_output=True, text=True)
    assert r.returncode != 0 and "static assertion failed" in r.stderr
