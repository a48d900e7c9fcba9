"""Depths whose metres overflow to infinity (a tiny depth scale and no upper
limit): a difference of two of them is NaN, which the filter's sums take in, so
such pixels come out 0 at every radius, the default 2 included, as in the
reference's arithmetic (depth_processing.hpp:71-115).  Against the oracle, bit
for bit."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1, 2, 3])
def test_infinite_metres(radius):
    rng = np.random.default_rng(radius)
    raw = rng.integers(0, 65536, (37, 45)).astype(np.uint16)
    raw[:, :6] = rng.integers(1, 40, (37, 6))  # finite metres, some beside infinite ones
    # raw / 3e-37 overflows from raw = 103 on
    options = dict(depth_scale=3e-37, min_depth=0.0, max_depth=float("inf"), bilateral_radius=radius)
    k = abi.Intrinsics(60.0, 60.0, 22.0, 18.0)
    pyr = kf.PyramidSource(kf.pipeline.default_depth_options(**options))
    pyr.build(raw, k)
    ref = ko.pyramid(raw, k, ko.depth_options(**options))[0]["depth"]
    assert np.array_equal(pyr.download_level(0)["depth"], ref)
    assert (ref == 0).any() and (ref != 0).any()
