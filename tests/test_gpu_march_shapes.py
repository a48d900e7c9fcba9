"""March CTAs of every accepted shape (1 to 64 threads), those that are not
whole warps included: a cooperative round hands samples to every lane of a warp.
Maps equal the default shape's, bit for bit, dense and sparse; the views' free
space and borders are where rounds turn cooperative.  The band march, which has
no such rounds, runs in the shape itself."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.fixture(scope="module", params=["dense", "sparse", "band march"])
def scene(request):
    seq = synthetic.make_sequence(seed=101, frames=2)
    pipeline = kf.Pipeline(kf.pipeline_config(
        (150, 130, 140), 0.03, (-2.25, -1.95, -0.5), 0.1, color=abi.KF_COLOR_NONE,
        storage=abi.KF_STORAGE_SPARSE if request.param == "sparse" else abi.KF_STORAGE_DENSE,
        integration_mode=abi.KF_INTEGRATION_BAND if request.param == "sparse" else abi.KF_INTEGRATION_FULL,
        raycast_backend=abi.KF_RAYCAST_BAND_MARCH if request.param == "band march" else abi.KF_RAYCAST_MARCH))
    for f in range(2):
        raw = seq.depth[f].copy()
        raw[:, 400:] = 0
        pipeline.integrate(raw, K640, ko.rigid_inverse(abi.rigid_from_matrix(seq.poses[f])))
    views = [(K640, 640, 480, np.array(seq.poses[1])), (abi.Intrinsics(330.0, 330.0, 200.0, 150.0), 401, 303, np.eye(4))]
    return pipeline, views, [pipeline.raycast(*v) for v in views]


@pytest.mark.parametrize("block", [(1, 1), (5, 5), (31, 1), (3, 11), (7, 9), (48, 1), (1, 63), (10, 5), (8, 8), (4, 8)])
def test_maps_do_not_depend_on_the_cta(scene, block):
    pipeline, views, expected = scene
    pipeline.set_launch_shapes(block, 148 * 48, raycast_lanes=(1, 1, 1))
    for view, want in zip(views, expected):
        got = pipeline.raycast(*view)
        for name in ("points", "normals", "colors"):
            a, b = getattr(got, name), getattr(want, name)
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (block, name)
    assert np.isfinite(expected[0].points).any()
