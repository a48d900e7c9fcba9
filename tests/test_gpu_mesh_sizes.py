"""The mesher's row pass (eight cells of a brick layer per lane, 32 bricks per
warp step) and its device normal fill against the oracle, element for element,
at extents whose rows end inside a brick, at a lane, at a warp step and past
one; and again on the same pipeline, whose working arrays then exist."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.fixture(scope="module")
def seq():
    return synthetic.make_sequence(seed=51, frames=2)


@pytest.mark.parametrize("res,voxel,policy", [
    ((2, 2, 2), abi.KF_VOXEL_FLOAT, abi.KF_CORNERS_SKIP_MISSING),
    ((9, 40, 33), abi.KF_VOXEL_FLOAT, abi.KF_CORNERS_SKIP_MISSING),
    ((64, 65, 66), abi.KF_VOXEL_QUANTIZED, abi.KF_CORNERS_REQUIRE_ALL),
    ((257, 30, 41), abi.KF_VOXEL_BF16, abi.KF_CORNERS_SKIP_MISSING),
    ((263, 24, 96), abi.KF_VOXEL_FLOAT, abi.KF_CORNERS_REQUIRE_ALL),
])
def test_mesh_matches_oracle(seq, res, voxel, policy):
    vs = 4.0 / max(res)
    origin, trunc = (-0.5 * res[0] * vs, -0.5 * res[1] * vs, 0.2), max(0.05, 3 * vs)
    gpu = kf.Pipeline(kf.pipeline_config(res, vs, origin, trunc, voxel=voxel, raycast_corner_policy=policy))
    assert gpu.extract_mesh()["positions"].size == 0  # nothing fused yet
    ref = ko.OracleVolume(res, vs, origin, trunc, voxel=voxel, color=True)
    for f in range(2):
        w2c = ko.rigid_inverse(abi.rigid_from_matrix(seq.poses[f]))
        normals = ko.pyramid(seq.depth[f], K640, ko.depth_options())[0]["normals"]
        gpu.integrate(seq.depth[f], K640, w2c, color=seq.color[f], normals=normals)
        ko.integrate(ref, seq.depth[f], K640, w2c, ko.integration_options(), abi.KF_RULE_ANGLE_WEIGHTED,
                     color=seq.color[f], normals_map=normals, threads=8)
        for min_weight in (0.0, 0.6):
            got, want = gpu.extract_mesh(min_weight), ko.marching_cubes(ref, min_weight)
            for name in ("positions", "normals", "colors", "triangles"):
                assert np.array_equal(got[name], want[name], equal_nan=got[name].dtype.kind == "f"), (f, min_weight, name)
    assert max(res) < 64 or got["triangles"].size > 0
