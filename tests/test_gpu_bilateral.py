"""The bilateral filter's staged tile and table exponential against the oracle,
bit for bit: radii whose staging spans one or several pixels per thread, a
radius past the staging's 48 KB (read directly), the pairwise weights of radius
2, sigmas that reach subnormal
and vanishing weights, and images smaller than a tile."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,radius,spatial,depth", [
    (97, 61, 1, 2.0, 0.08), (97, 61, 2, 2.0, 0.08), (33, 17, 2, 0.4, 0.004), (1, 5, 2, 3.0, 2.0), (65, 33, 7, 0.35, 0.01), (3, 2, 5, 4.0, 0.5), (70, 50, 28, 40.0, 4.0),
    (70, 50, 31, 9.0, 0.2),
])
def test_bilateral_matches_oracle(width, height, radius, spatial, depth):
    rng = np.random.default_rng(radius)
    raw = (5000 * (1.0 + 0.3 * rng.random((height, width)) + 0.02 * np.arange(width))).astype(np.uint16)
    raw[rng.random(raw.shape) < 0.1] = 0
    raw[:, width // 2:] += 9000
    options = dict(bilateral_radius=radius, bilateral_spatial_sigma=spatial, bilateral_depth_sigma=depth)
    k = abi.Intrinsics(60.0, 60.0, width / 2, height / 2)
    pyr = kf.PyramidSource(kf.pipeline.default_depth_options(**options))
    n = pyr.build(raw, k)
    ref = ko.pyramid(raw, k, ko.depth_options(**options))
    assert n == len(ref)
    for level in range(n):
        got = pyr.download_level(level)
        for name in ("depth", "vertices", "normals"):
            assert np.array_equal(got[name], ref[level][name], equal_nan=True), (level, name)
