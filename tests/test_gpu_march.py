"""The march's exact shortcuts on the GPU against the CPU oracle's plain march:
corner gathers across brick borders and at the volume's border, O(1) replays
of the ray-length additions over binade ends and half-way steps, cooperative
rounds, and cameras inside and outside the volume.  Maps are compared bit for
bit: every shortcut takes the plain march's samples."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.fixture(scope="module")
def seq():
    return synthetic.make_sequence(seed=11, frames=3, max_step_m=0.05, max_step_deg=3.0)


def same(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)


def pair(seq, res, vs, voxel=abi.KF_VOXEL_FLOAT, frames=2, **opts):
    origin = (-0.5 * res[0] * vs, -0.5 * res[1] * vs, -0.5)
    trunc = max(0.05, 3 * vs)
    gpu = kf.Pipeline(kf.pipeline_config(res, vs, origin, trunc, voxel=voxel, color=abi.KF_COLOR_NONE, **opts))
    ref = ko.OracleVolume(res, vs, origin, trunc, voxel=voxel)
    for f in range(frames):
        raw = seq.depth[f].copy()
        raw[:, 400:] = 0  # part of the view unobserved: mixed bricks along the frustum's sides
        normals = ko.pyramid(raw, K640, ko.depth_options())[0]["normals"]
        w2c = ko.rigid_inverse(abi.rigid_from_matrix(seq.poses[f]))
        gpu.integrate(raw, K640, w2c, normals=normals)
        ko.integrate(ref, raw, K640, w2c, ko.integration_options(), abi.KF_RULE_ANGLE_WEIGHTED, normals_map=normals,
                     threads=8)
    return gpu, ref


def turned(back, yaw):
    pose = np.eye(4)
    c, s = np.cos(yaw), np.sin(yaw)
    pose[:3, :3] = [[c, 0, s], [0, 1, 0], [-s, 0, c]]
    pose[2, 3] = -back
    return pose


@pytest.mark.parametrize("res,vs,scale,policy,voxel", [
    ((96, 80, 72), 0.04, 1.0, abi.KF_CORNERS_SKIP_MISSING, abi.KF_VOXEL_FLOAT),
    # the step lies halfway between two floats once the ray length passes 2
    ((120, 97, 133), 2.0 ** -5 + 2.0 ** -22, 1.0, abi.KF_CORNERS_SKIP_MISSING, abi.KF_VOXEL_FLOAT),
    ((65, 71, 79), 0.05, 0.37, abi.KF_CORNERS_REQUIRE_ALL, abi.KF_VOXEL_FLOAT),
    ((129, 128, 127), 0.03, 1.9, abi.KF_CORNERS_REQUIRE_ALL, abi.KF_VOXEL_BF16),
    ((7, 9, 8), 0.4, 0.25, abi.KF_CORNERS_SKIP_MISSING, abi.KF_VOXEL_QUANTIZED),
])
def test_march_matches_the_plain_march(seq, res, vs, scale, policy, voxel):
    gpu, ref = pair(seq, res, vs, voxel, raycast_corner_policy=policy, raycast_step_scale=scale)
    o = ko.raycast_options(corner_policy=policy, step_scale=scale)
    # widths of the three lane counts per ray (8, 4 and 1), odd extents
    for width, height, pose in ((131, 97, turned(0.0, 0.25)), (251, 189, turned(1.3, -0.4)), (401, 303, turned(0.1, 1.1))):
        k = abi.Intrinsics(0.8 * width, 0.8 * width, 0.5 * width, 0.5 * height)
        maps = gpu.raycast(k, width, height, pose)
        p, n, c = ko.raycast(ref, k, width, height, pose, o, threads=8)
        assert same(maps.points, p) and same(maps.normals, n) and same(maps.colors, c)
    assert np.isfinite(gpu.raycast(K640, 640, 480, np.eye(4)).points).any()
