"""The cells of a launch of the viscous least squares: each written once, by its
tile where it is in one, else by the block of its left-over group
(tests/visc_cells_check.cu, compiled with nvcc as host code; no GPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not os.path.exists(nvcc) and not shutil.which("nvcc"):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("visccells") / "visc_cells_check")
    subprocess.check_call([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "visc_cells_check.cu"), "-o", exe])
    return exe


@pytest.mark.parametrize("n,left", [(1, 1), (128, 0), (130, 3), (500, 60), (1000, 999), (4099, 40)])
def test_every_cell_is_written_once(check, n, left):
    rng = np.random.default_rng(n)
    own = np.sort(rng.permutation(n)[:left])  # cells that are in no tile
    tiled = np.ones(n, dtype=int)
    tiled[own] = 0
    cells = np.flatnonzero(tiled)
    ntile = -(-cells.size // 128)
    tcell = np.full(ntile * 128, -1)
    tcell[:cells.size] = cells
    ugrp = np.unique(own // 32)
    text = " ".join(str(v) for v in (n, ntile, ugrp.size, *tcell, *ugrp, *tiled))
    out = np.array(subprocess.run([check], input=text, capture_output=True, text=True, check=True).stdout.split(), int)
    assert np.array_equal(out, np.ones(2 * n, dtype=int))
