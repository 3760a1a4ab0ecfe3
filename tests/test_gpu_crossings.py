"""Crossing points of the mixed solver whose facets tie in FP32.  Paths of 50 m round at 4e-6 m
in FP32, and two facets (or a facet and the node between them) whose paths tie may cross
millimetres apart, so the choice is part of the result: the first facet in order (-x -y,
-x +y, +x -y, +x +y) with the smallest path, a facet whose minimum is the node having the
node's path.  The vectors were recorded from a solver that walks the four facets in that order;
half of them are such ties.  The FP64 final step leaves a chosen facet's crossing at 1e-12 m,
another choice shows above 1e-6 m."""
from pathlib import Path

import numpy as np
import pytest

import bsar

G = np.load(Path(__file__).parent / "golden" / "mixed_crossings.npz")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, len(G["a"])])
def test_tied_facets_keep_their_order(ctx, n):
    dem = bsar.DemArrays(G["x"], G["y"], G["z"])
    got = ctx.refraction_points(dem, G["a"][-n:], G["b"][-n:], 1.0, float(G["n2"]), solver="newton", precision="mixed")
    assert np.abs(got - G["crossing"][-n:]).max() <= 1e-9
