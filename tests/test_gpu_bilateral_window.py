"""The bilateral window is clipped to the image (depth_processing.hpp:79-82):
a radius at, past and far past the image's extent is every pixel of the image,
on both the staged and the direct path, against the oracle, bit for bit."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,radius", [
    (9, 7, 8), (9, 7, 27),             # staged: the window is the image
    (70, 50, 69), (70, 50, 70),        # direct, at and past the last pixel
    (70, 50, 1_000_000_000), (1, 1, 5), (3, 40, 1_000_000_000),
])
def test_window_is_clipped_to_the_image(width, height, radius):
    rng = np.random.default_rng(width + radius % 97)
    raw = (5000 * (1.0 + 0.3 * rng.random((height, width)))).astype(np.uint16)
    raw[rng.random(raw.shape) < 0.1] = 0
    options = dict(bilateral_spatial_sigma=20.0, bilateral_depth_sigma=0.2)
    k = abi.Intrinsics(60.0, 60.0, width / 2, height / 2)
    pyr = kf.PyramidSource(kf.pipeline.default_depth_options(bilateral_radius=radius, **options))
    pyr.build(raw, k)
    # the oracle's own window arithmetic is 32-bit: the same window, from the largest radius that matters
    ref = ko.pyramid(raw, k, ko.depth_options(bilateral_radius=min(radius, max(width, height)), **options))
    assert np.array_equal(pyr.download_level(0)["depth"], ref[0]["depth"])
