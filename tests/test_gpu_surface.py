"""The mixed image of voxels within a node spacing of the surface against the FP64 Newton image,
one pulse at a time so that every voxel is one pair of solves.  The solvers' undamped steps
cycle there, and the facet that wins follows the order of the facets; FP32 paths that tie within
4e-6 m choose otherwise in a small share of the voxels, which is recorded: 607 of 1.08 million
voxels more than 1 % off, twice as many when a facet whose steps end back on the node is taken
before the facets that keep it."""
import numpy as np
import pytest

import bsar
from bsar import scene as S

pytestmark = pytest.mark.gpu


def test_mixed_follows_the_solvers_facets(ctx):
    off = total = 0
    for seed in range(3):
        sc = S.make_scene(S.scaled(S.config_spec(2), n_pulses=1, n_samples=4096, n_scatterers=2, nx=300, ny=300, nz=1,
                                   seed=seed), with_raw=False)
        rng = np.random.default_rng(5)
        sc.raw = rng.normal(size=(1, 4096)) + 1j * rng.normal(size=(1, 4096))
        sid = bsar.upload_scene(ctx, sc)
        gz = np.array([-0.5, -0.2, 0.0, 0.3])
        try:
            mixed, fp64 = (ctx.backproject(sid, sc.gx, sc.gy, gz, solver="newton", legs="per_pulse", precision=p)
                           for p in ("mixed", "fp64"))
        finally:
            ctx.scene_release(sid)
        off += int((np.abs(mixed - fp64) > 1e-2 * np.abs(fp64).mean()).sum())
        total += fp64.size
    assert off <= 8e-4 * total
