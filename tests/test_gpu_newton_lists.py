"""The FP64 Newton back-projection on candidate lists (k_newton.cu) against the oracle's FP64
Newton image, rel-L2 <= 1e-9, where its branches differ: short and long lists, no list,
windows cut by the DEM's border, equal indices and a lower one below ground, an exactly flat
DEM, few pulses far apart, and the warps-per-voxel splits (few and many pulses, grids with
remainders)."""
import numpy as np
import pytest

import bsar
from bsar import scene as S
import oracle as O

from conftest import rel_l2

pytestmark = pytest.mark.gpu

CASES = {
    "rough": dict(nx=7, ny=9, nz=3),
    "coarse voxels": dict(nx=5, ny=9, nz=2, dxy=0.5, dz=0.4),
    "fine dem": dict(nx=4, ny=5, nz=2, dem_d=0.08, dem_n=300),
    "dem border": dict(nx=6, ny=7, nz=2, dxy=0.3, dem_n=14),
    "equal indices": dict(nx=5, ny=6, nz=2, eps_r=1.0),
    "lower index": dict(nx=5, ny=6, nz=2, eps_r=0.5),
    "flat dem": dict(nx=5, ny=5, nz=3, dxy=0.27, dem_sigma=0.0, dem_kind="plane"),
    "smooth dem": dict(nx=5, ny=6, nz=3, dem_sigma=0.002, dem_kind="plane"),
    "pulses apart": dict(nx=5, ny=6, nz=2, n_pulses=9),
    "many pulses": dict(nx=3, ny=3, nz=1, n_pulses=1100),
    "eight warps": dict(nx=3, ny=5, nz=1, n_pulses=300),
    "one pulse": dict(nx=3, ny=5, nz=1, n_pulses=1),
}


@pytest.mark.parametrize("name", CASES)
def test_newton_image_matches_the_oracle(ctx, oracle, name):
    spec = S.scaled(S.config_spec(2), **{**dict(n_pulses=50, n_samples=4096, n_scatterers=2), **CASES[name]})
    sc = S.make_scene(spec, with_raw=False)
    rng = np.random.default_rng(5)
    sc.raw = rng.normal(size=(spec.n_pulses, 4096)) + 1j * rng.normal(size=(spec.n_pulses, 4096))
    sid = bsar.upload_scene(ctx, sc)
    try:
        img = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, solver="newton", legs="per_pulse", precision="fp64")
    finally:
        ctx.scene_release(sid)
    rc = oracle.spline_upsample(oracle.fft_correlate(sc.raw, sc.reference), spec.upsample)
    want = oracle.backproject(O.Dem(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, rc, sc.gx, sc.gy, sc.gz, spec.n1, spec.n2,
                              3e8, sc.fs_eff, sc.lam, legs="per", solver="newton",
                              search_nodes=S.search_nodes_for(sc.x_vec, sc.y_vec))
    assert np.abs(want).max() > 0
    assert rel_l2(img, want) <= 1e-9


@pytest.mark.parametrize("height", [300.0, 2000.0, 8000.0, -9000.3])
@pytest.mark.parametrize("n_pulses", [1, 50])
def test_raised_terrain(ctx, oracle, height, n_pulses):
    """Terrain, antennas and voxels far above or below zero, where FP32 heights round at up to
    half a millimetre: the image is still the oracle's."""
    spec = S.scaled(S.config_spec(2), n_pulses=n_pulses, n_samples=4096, n_scatterers=2, nx=9, ny=10, nz=2)
    sc = S.make_scene(spec, with_raw=False)
    rng = np.random.default_rng(5)
    sc.raw = rng.normal(size=(n_pulses, 4096)) + 1j * rng.normal(size=(n_pulses, 4096))
    up = np.array([0.0, 0.0, height])
    sc.z, sc.tx, sc.rx, sc.gz = sc.z + height, sc.tx + up, sc.rx + up, sc.gz + height
    sid = bsar.upload_scene(ctx, sc)
    try:
        img = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, solver="newton", legs="per_pulse", precision="fp64")
    finally:
        ctx.scene_release(sid)
    rc = oracle.spline_upsample(oracle.fft_correlate(sc.raw, sc.reference), spec.upsample)
    want = oracle.backproject(O.Dem(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, rc, sc.gx, sc.gy, sc.gz, spec.n1, spec.n2,
                              3e8, sc.fs_eff, sc.lam, legs="per", solver="newton",
                              search_nodes=S.search_nodes_for(sc.x_vec, sc.y_vec))
    assert rel_l2(img, want) <= 1e-9


@pytest.mark.parametrize("n_pulses", [1, 7, 50])
def test_large_grid_has_the_small_grids_image(ctx, n_pulses):
    """114000 voxels take two warps per 32 voxels, their first three x planes four: both within
    1e-9 of the oracle, so within 2e-9 of each other."""
    spec = S.scaled(S.config_spec(2), n_pulses=n_pulses, n_samples=4096, n_scatterers=2, nx=76, ny=50, nz=30, dxy=0.02)
    sc = S.make_scene(spec, with_raw=False)
    rng = np.random.default_rng(6)
    sc.raw = rng.normal(size=(n_pulses, 4096)) + 1j * rng.normal(size=(n_pulses, 4096))
    sid = bsar.upload_scene(ctx, sc)
    form = dict(solver="newton", legs="per_pulse", precision="fp64")
    try:
        big = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, **form)
        small = ctx.backproject(sid, sc.gx[:3], sc.gy, sc.gz, **form)
    finally:
        ctx.scene_release(sid)
    assert np.abs(small).max() > 0
    assert rel_l2(big[:3], small) <= 2e-9


@pytest.mark.parametrize("n_pulses", [1, 17, 50, 300, 1100])
def test_a_voxel_has_one_value_in_every_grid(ctx, n_pulses):
    """Grids that take 4 to 16 warps per 32 voxels, ranges of them and single voxels: the same
    bits, since the order of a voxel's sum follows the pulses alone."""
    spec = S.scaled(S.config_spec(2), n_pulses=n_pulses, n_samples=4096, n_scatterers=2, nx=61, ny=63, nz=31, dxy=0.02)
    sc = S.make_scene(spec, with_raw=False)
    rng = np.random.default_rng(6)
    sc.raw = rng.normal(size=(n_pulses, 4096)) + 1j * rng.normal(size=(n_pulses, 4096))
    sid = bsar.upload_scene(ctx, sc)
    form = dict(solver="newton", legs="per_pulse", precision="fp64")
    try:
        big = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, **form)
        for x, y, z in ((slice(0, 61), slice(0, 63), slice(3, 4)), (slice(5, 9), slice(7, 16), slice(2, 5)),
                        (slice(0, 61), slice(0, 63), slice(0, 13)), (slice(60, 61), slice(2, 3), slice(30, 31))):
            small = ctx.backproject(sid, sc.gx[x], sc.gy[y], sc.gz[z], **form)
            assert np.array_equal(small, big[x, y, z])
        part = ctx.backproject_range(sid, sc.gx, sc.gy, sc.gz, 1001, 5002, **form)
    finally:
        ctx.scene_release(sid)
    flat = np.arange(1001, 1001 + 5002)                      # z -> x -> y
    at = (flat // 63) % 61, flat % 63, flat // (61 * 63)
    assert np.array_equal(part[at], big[at])


@pytest.mark.parametrize("seed,voxel", [(6, (62, 0, 22)), (6, (65, 25, 16)), (6, (56, 35, 3)), (3, (7, 7, 21)),
                                        (26, (34, 40, 0))])
def test_every_open_facet_is_polished(ctx, oracle, seed, voxel):
    """Voxels with a crossing whose edge minimum three Newton steps reach from one of the edge's
    two facets only.  Paths of 50 m round at 7e-15 m, 1.5e-13 rad of phase; 1e-11 leaves room for
    some sixty roundings per path, and a facet left out shows as 1e-7."""
    spec = S.scaled(S.config_spec(2), n_pulses=256, n_samples=4096, n_scatterers=2, seed=seed, nx=81, ny=77, nz=24,
                    dem_sigma=0.5, eps_r=3.0)
    sc = S.make_scene(spec, with_raw=False)
    rng = np.random.default_rng(5)
    sc.raw = rng.normal(size=(256, 4096)) + 1j * rng.normal(size=(256, 4096))
    gx, gy, gz = (g[i:i + 1] for g, i in zip((sc.gx, sc.gy, sc.gz), voxel))
    sid = bsar.upload_scene(ctx, sc)
    try:
        img = ctx.backproject(sid, gx, gy, gz, solver="newton", legs="per_pulse", precision="fp64")
    finally:
        ctx.scene_release(sid)
    rc = oracle.spline_upsample(oracle.fft_correlate(sc.raw, sc.reference), spec.upsample)
    want = oracle.backproject(O.Dem(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, rc, gx, gy, gz, spec.n1, spec.n2, 3e8,
                              sc.fs_eff, sc.lam, legs="per", solver="newton",
                              search_nodes=S.search_nodes_for(sc.x_vec, sc.y_vec))
    assert rel_l2(img, want) <= 1e-11


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_voxels_at_the_surface(ctx, oracle, seed):
    """Undamped Newton steps cycle between a facet's corners when the voxel lies within a node
    spacing of the surface: a facet may end above its node or back on it, and the image follows
    the solver's choice among such facets.  Rounding grows with the steps: single paths differ
    by up to 7e-11 of a radian, a facet chosen otherwise by up to a whole turn."""
    spec = S.scaled(S.config_spec(2), n_pulses=40, n_samples=4096, n_scatterers=2, seed=seed, nx=31, ny=30, nz=1, dxy=0.1)
    sc = S.make_scene(spec, with_raw=False)
    rng = np.random.default_rng(5)
    sc.raw = rng.normal(size=(40, 4096)) + 1j * rng.normal(size=(40, 4096))
    gz = np.array([-0.5, -0.2, 0.0, 0.3])
    sid = bsar.upload_scene(ctx, sc)
    try:
        img = ctx.backproject(sid, sc.gx, sc.gy, gz, solver="newton", legs="per_pulse", precision="fp64")
    finally:
        ctx.scene_release(sid)
    rc = oracle.spline_upsample(oracle.fft_correlate(sc.raw, sc.reference), spec.upsample)
    want = oracle.backproject(O.Dem(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, rc, sc.gx, sc.gy, gz, spec.n1, spec.n2, 3e8,
                              sc.fs_eff, sc.lam, legs="per", solver="newton",
                              search_nodes=S.search_nodes_for(sc.x_vec, sc.y_vec))
    assert rel_l2(img, want) <= 1e-9
