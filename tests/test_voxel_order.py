"""The order in which the mixed kernel takes the voxels of whole z-planes (compact_voxel,
kernels.hpp): every voxel once, and consecutive voxels next to each other, so that the 32
voxels of a warp form a compact block whatever the grid's remainders are."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = tmp_path_factory.mktemp("order") / "voxel_order"
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", f"-I{ROOT / 'c-_bistatic_sar_b200' / 'csrc'}",
                    f"-I{ROOT / 'include'}", "-I/usr/local/cuda/include",
                    str(Path(__file__).parent / "compat" / "voxel_order_driver.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("n", [(1, 1, 1), (3, 5, 1), (4, 8, 2), (5, 7, 3), (17, 1, 4), (1, 40, 3), (41, 41, 21),
                               (16, 33, 5)])
def test_every_voxel_once_and_neighbours_together(driver, n):
    out = subprocess.run([str(driver), *map(str, n)], check=True, capture_output=True, text=True).stdout
    v = np.array(out.split(), dtype=np.int64).reshape(-1, 3)
    flat = (v[:, 0] * n[1] + v[:, 1]) * n[2] + v[:, 2]
    assert np.array_equal(np.sort(flat), np.arange(n[0] * n[1] * n[2]))
    # one step never leaves the neighbouring block of 4 x 1 x 2 voxels
    assert (np.abs(np.diff(v, axis=0)) <= np.array([7, 1, 3])).all()
