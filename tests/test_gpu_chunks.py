"""Pulse chunks of small grids where their sums have no room (a tight budget, the no-alloc
scratch): the chunks run one after the other and add to the image, in the order and with the
bits of the chunks that run side by side, so an image does not depend on the memory that
happens to be free."""
import numpy as np
import pytest

import bsar
from bsar import scene as S

pytestmark = pytest.mark.gpu

HOW = dict(solver="newton", legs="per_pulse")


def _scene(n_pulses=300, n_samples=256, **kw):
    sc = S.make_scene(S.scaled(S.config_spec(2), **{**dict(n_pulses=n_pulses, n_samples=4096, n_scatterers=2, nx=33, ny=35,
                                                           nz=21, dxy=0.03), **kw}), with_raw=False)
    rng = np.random.default_rng(3)
    data = rng.normal(size=(n_pulses, n_samples)) + 1j * rng.normal(size=(n_pulses, n_samples))
    return sc, data


def _upload(ctx, sc, data):
    # 256 samples cover the scene's delays: 60 to 130 m of path at 0.6 GHz after upsampling
    return ctx.scene_upload(bsar.DemArrays(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, data, kind="compressed", upsample=2,
                            n1=1.0, n2=6.0 ** 0.5, c=3e8, fc=1e9, fs=0.3e9)


@pytest.mark.parametrize("dem", [dict(), dict(dem_d=0.125, dem_n=256), dict(dem_d=0.2)])
@pytest.mark.parametrize("precision", ["mixed", "mixed_fp16"])
def test_tight_budget_has_the_same_bits(ctx, precision, dem):
    sc, data = _scene(**dem)
    axes = sc.gx, sc.gy, sc.gz
    nv = sc.gx.size * sc.gy.size * sc.gz.size
    sid = _upload(ctx, sc, data)
    before = ctx.bytes_in_use
    ctx.scene_compress(sid, precision)
    n = ctx.launches
    want = ctx.backproject(sid, *axes, precision=precision, **HOW)
    side_by_side = ctx.launches - n
    part = ctx.backproject_range(sid, *axes, 1001, 9002, precision=precision, **HOW)
    ctx.scene_release(sid)
    assert np.abs(want).min() > 0
    # room for the scene and the image, not for K >= 2 more of them
    with bsar.Context(0, hbm_budget_bytes=(before - ctx.bytes_in_use) + 16 * 2 * data.size + 2 * 16 * nv) as tight:
        sid = _upload(tight, sc, data)
        tight.scene_compress(sid, precision)
        for _ in range(2):
            n = tight.launches
            assert np.array_equal(tight.backproject(sid, *axes, precision=precision, **HOW), want)
            assert tight.launches - n > side_by_side                   # a launch per chunk
        assert np.array_equal(tight.backproject_range(sid, *axes, 1001, 9002, precision=precision, **HOW), part)


def test_noalloc_scratch_without_room_has_the_same_bits(ctx):
    """1.25 million pulses' anchors leave 2 MB of the scratch: the image fits, its chunks do not."""
    sc, data = _scene(n_pulses=1_250_000, n_samples=8, nx=27, ny=27, nz=26)
    sid = ctx.scene_upload(bsar.DemArrays(sc.x_vec, sc.y_vec, sc.z), sc.tx, sc.rx, data, kind="compressed", upsample=1,
                           n1=1.0, n2=6.0 ** 0.5, c=3e8, fc=1e9, fs=1e7)
    try:
        ctx.scene_compress(sid, "mixed")
        want = ctx.backproject(sid, sc.gx, sc.gy, sc.gz, precision="mixed", **HOW)
        got = ctx.backproject_mixed_noalloc(sid, sc.gx, sc.gy, sc.gz)
    finally:
        ctx.scene_release(sid)
    assert np.abs(want).min() > 0
    assert np.array_equal(got, want)
