"""The mixed kernel's candidate lists (a node scan shared by a warp's voxels and a block of
pulses) against the scan that ranks every node of every window (exhaustive=True): the image
must be the same bit for bit, over the geometries where the lists take other branches:
long lists and no list (coarse voxels, fine DEMs), windows cut by the DEM's border or moving
over the block (nodes outside some window), equal indices (the antenna is the lower endpoint
of one leg), a lower index below ground, exact ties (a flat DEM), pulses far apart, low
antennas, voxels at the surface, and grids with remainders in every axis."""
import numpy as np
import pytest

import bsar
from bsar import scene as S

pytestmark = pytest.mark.gpu

# name: (scene fields, antenna shift in z, z axis or None, search radius)
CASES = {
    "coarse voxels": (dict(nx=9, ny=17, nz=3, dxy=0.5, dz=0.4), 0.0, None, 0.0),
    "fine dem": (dict(nx=10, ny=13, nz=3, dem_d=0.06, dem_n=400), 0.0, None, 0.0),
    "wide window": (dict(nx=6, ny=9, nz=2, dem_d=0.125, dem_n=300), 0.0, None, 4.0),
    "one-node window": (dict(nx=8, ny=9, nz=2, dem_d=2.0, dem_n=40), 0.0, None, 0.0),
    "dem border": (dict(nx=12, ny=11, nz=3, dxy=0.2, dem_n=14), 0.0, None, 0.0),
    "border, wide": (dict(nx=12, ny=11, nz=3, dxy=0.2, dem_d=0.125, dem_n=30), 0.0, None, 0.0),
    "equal indices": (dict(nx=9, ny=10, nz=3, eps_r=1.0), 0.0, None, 0.0),
    "lower index": (dict(nx=9, ny=10, nz=3, eps_r=0.5), 0.0, None, 0.0),
    "flat dem": (dict(nx=9, ny=9, nz=3, dxy=0.25, dem_sigma=0.0, dem_kind="plane"), 0.0, None, 0.0),
    "smooth dem": (dict(nx=13, ny=14, nz=3, dem_sigma=0.002, dem_kind="plane"), 0.0, None, 0.0),
    "pulses apart": (dict(nx=9, ny=10, nz=3, n_pulses=9), 0.0, None, 0.0),
    "low antennas": (dict(nx=9, ny=10, nz=3, n_pulses=60), -27.5, None, 0.0),
    "surface voxels": (dict(nx=13, ny=10, nz=4), 0.0, np.array([-0.5, -0.2, 0.0, 0.3]), 0.0),
    "single voxel": (dict(nx=1, ny=1, nz=1, n_scatterers=1), 0.0, None, 0.0),
    "rows": (dict(nx=3, ny=45, nz=1), 0.0, None, 0.0),
    "columns": (dict(nx=45, ny=1, nz=3), 0.0, None, 0.0),
}


@pytest.mark.parametrize("precision", ["mixed", "mixed_fp16"])
@pytest.mark.parametrize("name", CASES)
def test_lists_give_the_exhaustive_image(ctx, name, precision):
    _lists_equal_exhaustive(ctx, name, precision)


@pytest.mark.parametrize("name", CASES)
def test_fp64_lists_give_the_exhaustive_image(ctx, name):
    """The same of the FP64 Newton kernel, whose lists are bounded in FP32."""
    _lists_equal_exhaustive(ctx, name, "fp64")


def _lists_equal_exhaustive(ctx, name, precision):
    kw, dz, gz, radius = CASES[name]
    sc = S.make_scene(S.scaled(S.config_spec(2), **{**dict(n_pulses=70, n_samples=4096, n_scatterers=3), **kw}),
                      with_raw=False)
    sc.tx = sc.tx + np.array([0.0, 0.0, dz])
    sc.rx = sc.rx + np.array([0.0, 0.0, dz])
    rng = np.random.default_rng(11)
    sc.raw = rng.normal(size=(len(sc.tx), 4096)) + 1j * rng.normal(size=(len(sc.tx), 4096))
    z = sc.gz if gz is None else gz
    how = dict(solver="newton", legs="per_pulse", precision=precision, search_radius_m=radius)
    sid = bsar.upload_scene(ctx, sc)
    try:
        full = ctx.backproject(sid, sc.gx, sc.gy, z, exhaustive=True, **how)
        lists = ctx.backproject(sid, sc.gx, sc.gy, z, **how)
    finally:
        ctx.scene_release(sid)
    assert np.abs(full).max() > 0
    assert np.array_equal(lists, full)


# name: (scale of all lengths, height added to everything, scene fields, voxel clusters)
PLACES = {
    "terrain at 300 m": (1, 300.0, {}, False),
    "terrain at 2000 m": (1, 2000.0, {}, False),
    "terrain at 8000 m": (1, 8000.0, {}, False),
    "terrain at -9000 m": (1, -9000.3, {}, False),
    "smooth at 8000 m": (1, 8000.0, dict(dem_sigma=0.002, dem_kind="plane"), False),
    "one pulse at 8000 m": (1, 8000.0, dict(n_pulses=1), True),
    "one pulse": (1, 0.0, dict(n_pulses=1), True),
    "paths of 1 km": (20, 0.0, {}, False),
    "paths of 5 km": (100, 0.0, {}, False),
    "paths of 5 km, flat": (100, 0.0, dict(dem_sigma=0.03), False),
    "paths of 15 km": (300, 0.0, {}, False),
    "dem of 1.5 km": (1, 0.0, dict(dem_d=0.37, dem_n=4000), False),
}


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("name", PLACES)
def test_lists_far_from_the_origin(ctx, name, precision):
    """Heights, coordinates and paths whose FP32 rounding is far above that of the scenes above;
    clusters of voxels micrometres apart and one pulse leave the lists' bounds no slack."""
    k, shift, kw, clusters = PLACES[name]
    spec = S.scaled(S.config_spec(2), **{**dict(n_pulses=120, n_samples=4096, n_scatterers=2, nx=24, ny=23, nz=4), **kw})
    sc = S.make_scene(spec, with_raw=False)
    up = np.array([0.0, 0.0, shift])
    rng = np.random.default_rng(5)
    data = rng.normal(size=(spec.n_pulses, 4096)) + 1j * rng.normal(size=(spec.n_pulses, 4096))
    axes = [sc.gx, sc.gy, sc.gz]
    if clusters:
        c = np.arange(4) * 1e-6
        axes = [(np.linspace(17, 23, 60)[:, None] + c).ravel(), (np.linspace(-3, 3, 60)[:, None] + c).ravel(), -5.0 + c[:2]]
    dem = bsar.DemArrays(sc.x_vec * k, sc.y_vec * k, sc.z * k + shift)
    sid = ctx.scene_upload(dem, sc.tx * k + up, sc.rx * k + up, data, kind="compressed", upsample=2, n1=1.0, n2=6.0 ** 0.5,
                           c=3e8, fc=1e9 / k, fs=1.92e9 / k)
    how = dict(solver="newton", legs="per_pulse", precision=precision, search_radius_m=1.5 * k)
    try:
        full = ctx.backproject(sid, axes[0] * k, axes[1] * k, axes[2] * k + shift, exhaustive=True, **how)
        lists = ctx.backproject(sid, axes[0] * k, axes[1] * k, axes[2] * k + shift, **how)
    finally:
        ctx.scene_release(sid)
    assert np.abs(full).min() > 0
    assert np.array_equal(lists, full)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("scene", [dict(dem_d=0.1, dem_n=400), dict(dxy=0.2, dz=0.3), dict(dxy=0.2, dem_n=14)])
@pytest.mark.parametrize("n1,n2", [(-1.0, 8.0), (-0.3, 2.0), (8.0, -0.1), (0.0, 2.0), (2.0, 0.0), (1e-50, 2.0)])
def test_indices_without_lists(ctx, n1, n2, scene, precision):
    """Any finite index is accepted; the lists' bounds hold for positive ones only."""
    sc = S.make_scene(S.scaled(S.config_spec(2), **{**dict(n_pulses=100, n_samples=4096, n_scatterers=2, nx=25, ny=26, nz=3),
                                                    **scene}), with_raw=False)
    rng = np.random.default_rng(5)
    data = rng.normal(size=(100, 4096)) + 1j * rng.normal(size=(100, 4096))
    sid = ctx.scene_upload(bsar.DemArrays(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, data, kind="compressed", upsample=2, n1=n1,
                           n2=n2, c=3e8, fc=1e9, fs=1.92e9)
    how = dict(solver="newton", legs="per_pulse", precision=precision)
    try:
        full = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, exhaustive=True, **how)
        lists = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, **how)
    finally:
        ctx.scene_release(sid)
    assert np.abs(full).max() > 0
    assert np.array_equal(lists, full)
