"""The Fermat solvers' other shapes against the ones they stand in for: a warp per solve
against a thread per solve (bit for bit), and the back-projection's grid search behind its
FP32 filter against the oracle, rel-L2 <= 1e-11, on DEMs where the filter's branches differ:
rough, smooth and exactly flat ones (ties), steps, a DEM much smaller than the search, large
heights, one at a search point's edge, and axes that are not evenly spaced (no filter)."""
import numpy as np
import pytest

import bsar
from bsar import scene as S
import oracle as O

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _points(n, rng):
    a = np.stack([rng.uniform(-15, 15, n), rng.uniform(-15, 15, n), np.full(n, 30.0)], axis=1)
    b = np.stack([20 + rng.uniform(-4, 4, n), rng.uniform(-4, 4, n), rng.uniform(-7, -2, n)], axis=1)
    return a, b


@pytest.mark.parametrize("solver", ["grid", "newton"])
@pytest.mark.parametrize("kind", ["plane", "fbm", "flat"])
def test_warp_solves_equal_thread_solves(ctx, solver, kind):
    spec = S.scaled(S.config_spec(2), dem_kind="plane" if kind == "flat" else kind,
                    dem_sigma={"plane": 0.05, "fbm": 0.4, "flat": 0.0}[kind], dem_n=65)
    x, y, z = S.make_dem(spec, np.random.default_rng(3))
    dem = bsar.DemArrays(x, y, z)
    a, b = _points(20000, np.random.default_rng(4))          # a thread per solve
    few = ctx.refraction_points(dem, a[:333], b[:333], 1.0, 2.0, solver=solver)
    many = ctx.refraction_points(dem, a, b, 1.0, 2.0, solver=solver)
    assert np.array_equal(few, many[:333])
    one = ctx.refraction_points(dem, a[:1], b[:1], 1.0, 2.0, solver=solver)
    assert np.array_equal(one, many[:1])
    # the per-voxel function: a warp per pulse and leg, and a thread per pulse
    P = b[0]
    few = ctx.slant_range_fermat(dem, a[:65], a[:65] + [5.0, 0, 0], P, 1.0, 2.0, solver=solver, reflection=True)
    many = ctx.slant_range_fermat(dem, a, a + [5.0, 0, 0], P, 1.0, 2.0, solver=solver, reflection=True)
    assert np.array_equal(few[0], many[0][:, :65])
    assert all(np.array_equal(f, m[:65]) for f, m in zip(few[1:], many[1:]))


def _dem(name):
    x = 20.0 + (np.arange(48) - 23.5) * 0.5
    y = (np.arange(40) - 19.5) * 0.5
    rng = np.random.default_rng(8)
    z = rng.normal(0, 0.05, (40, 48))
    if name == "rough":
        z = rng.normal(0, 0.6, (40, 48))
    elif name == "flat":
        z[:] = 0.0
    elif name == "steps":
        z[:, 24:] += 2.0
        z[20:] -= 1.0
    elif name == "small":
        x, y, z = x[22:26], y[18:21], z[18:21, 22:26]
    elif name == "two by two":
        x, y, z = x[[0, 47]], y[[0, 39]], z[:2, :2]
    elif name == "uneven":
        x = x + 0.1 * np.sin(np.arange(48))
    elif name == "at a search point":
        x = x - x[0] + 20.0            # the first axis value on the level's centre column
    return x, y, z


@pytest.mark.parametrize("legs", ["mean", "per_pulse"])
@pytest.mark.parametrize("name", ["plane", "rough", "flat", "steps", "small", "two by two", "uneven",
                                  "at a search point", "high"])
def test_filtered_grid_search_image(ctx, oracle, name, legs):
    x, y, z = _dem(name)
    spec = S.scaled(S.config_spec(1), n_pulses=45, nx=4, ny=3, nz=2, dxy=0.6, dz=0.7)
    sc = S.make_scene(spec, with_raw=False)
    tx, rx, gz = sc.tx, sc.rx, sc.gz
    if name == "high":                  # terrain at 2000 m
        z, gz = z + 2000.0, gz + 2000.0
        tx, rx = tx + [0, 0, 2000.0], rx + [0, 0, 2000.0]
    rng = np.random.default_rng(6)
    data = rng.normal(size=(45, 1024)) + 1j * rng.normal(size=(45, 1024))
    dem = bsar.DemArrays(x, y, z)
    kw = dict(upsample=4, n1=1.0, n2=2.0, c=3e8, fc=1e9, fs=1.2e9)
    sid = ctx.scene_upload(dem, tx, rx, data, kind="compressed", **kw)
    try:
        img = ctx.backproject(sid, sc.gx, sc.gy, gz, solver="grid", legs=legs, precision="fp64")
    finally:
        ctx.scene_release(sid)
    want = oracle.backproject(O.Dem(x, y, z), tx, rx, oracle.spline_upsample(data, 4), sc.gx, sc.gy, gz, 1.0, 2.0, 3e8,
                              sc.fs_eff, sc.lam, legs="mean" if legs == "mean" else "per", solver="grid")
    assert np.abs(want).max() > 0
    assert rel_l2(img, want) <= 1e-11


@pytest.mark.parametrize("value,share,seed", [(-9999.0, 0.2, 0), (-9999.0, 0.2, 1), (-32768.0, 0.02, 2),
                                              (-32768.0, 0.2, 3), (1e4, 0.2, 0), (1e4, 0.2, 4), (3000.0, 0.2, 5),
                                              (1e6, 0.2, 0), (3e38, 0.02, 1), (1e39, 0.02, 2), (-1e39, 0.2, 3)])
def test_filtered_grid_search_beside_outliers(ctx, oracle, value, share, seed):
    """No-data values and cliffs beside the terrain: the FP32 height of a point in such a cell
    is off by far more than its own magnitude says."""
    x, y, _ = _dem("plane")
    rng = np.random.default_rng([seed, int(100 * share), int(min(abs(value), 1e6))])
    z = rng.normal(0, 0.05, (40, 48))
    out = rng.random(z.shape) < share
    z[out] = value * (1 + 1e-3 * rng.normal(size=out.sum()))
    n = 64
    s = np.arange(n) / (n - 1)
    th = 6 * np.pi * s
    tx = np.stack([15 * (1 - s) * np.cos(th), 15 * (1 - s) * np.sin(th), np.full(n, 30.0)], 1)
    rx = tx + [5.0, 0.0, 0.0]
    axes = 20 + np.arange(8) * 0.37, -1 + np.arange(8) * 0.31, np.array([-6.0, -4.5, -3.0, -1.5])
    data = rng.normal(size=(n, 1024)) + 1j * rng.normal(size=(n, 1024))
    sid = ctx.scene_upload(bsar.DemArrays(x, y, z), tx, rx, data, kind="compressed", upsample=4, n1=1.0, n2=2.0, c=3e8,
                           fc=1e9, fs=1.2e9)
    try:
        img = ctx.backproject(sid, *axes, solver="grid", legs="per_pulse", precision="fp64")
    finally:
        ctx.scene_release(sid)
    want = oracle.backproject(O.Dem(x, y, z), tx, rx, oracle.spline_upsample(data, 4), *axes, 1.0, 2.0, 3e8, 4.8e9, 0.3,
                              legs="per", solver="grid")
    assert np.abs(want).max() > 0
    assert rel_l2(img, want) <= 1e-11
