"""The sparse march's shortcuts against the CPU oracle's plain march over the
dense volume that the sparse store stands for, bit for bit: block counts that do
not divide by the null cells' 4 and 16 blocks (partial cells at the border),
cells of either size crossed whole, cameras inside, at the border of and outside
the domain, each lane count per ray, and both corner rules."""

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.fixture(scope="module")
def seq():
    return synthetic.make_sequence(seed=81, frames=2, max_step_m=0.05, max_step_deg=3.0)


def same(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)


def turned(back, yaw, side=0.0):
    pose = np.eye(4)
    c, s = np.cos(yaw), np.sin(yaw)
    pose[:3, :3] = [[c, 0, s], [0, 1, 0], [-s, 0, c]]
    pose[:3, 3] = side, 0.0, -back
    return pose


@pytest.mark.parametrize("res,vs,scale,policy,voxel,cell_normals", [
    ((300, 173, 211), 0.02, 1.0, abi.KF_CORNERS_SKIP_MISSING, abi.KF_VOXEL_FLOAT, 0),
    ((65, 71, 523), 0.011, 0.6, abi.KF_CORNERS_REQUIRE_ALL, abi.KF_VOXEL_BF16, 1),
    ((521, 392, 401), 0.01, 1.0, abi.KF_CORNERS_SKIP_MISSING, abi.KF_VOXEL_BF16, 0),
    ((137, 129, 143), 0.04, 1.7, abi.KF_CORNERS_REQUIRE_ALL, abi.KF_VOXEL_QUANTIZED, 0),
    ((7, 9, 8), 0.4, 0.25, abi.KF_CORNERS_SKIP_MISSING, abi.KF_VOXEL_FLOAT, 0),
])
def test_sparse_march_matches_the_plain_march(seq, res, vs, scale, policy, voxel, cell_normals):
    origin = (-0.5 * res[0] * vs, -0.5 * res[1] * vs, -0.5)
    trunc = max(0.05, 3 * vs)
    blocks = int(np.prod([-(-r // 8) for r in res]))
    gpu = kf.Pipeline(kf.pipeline_config(
        res, vs, origin, trunc, voxel=voxel, color=abi.KF_COLOR_NONE, storage=abi.KF_STORAGE_SPARSE,
        integration_mode=abi.KF_INTEGRATION_BAND, sparse_block_capacity=blocks, raycast_corner_policy=policy,
        raycast_step_scale=scale, raycast_cell_gradient_normals=cell_normals))
    ref = ko.OracleVolume(res, vs, origin, trunc, voxel=voxel, sparse=True, capacity=blocks)
    for f in range(2):
        raw = seq.depth[f].copy()
        raw[:, 380:] = 0  # part of the view unobserved
        w2c = ko.rigid_inverse(abi.rigid_from_matrix(seq.poses[f]))
        gpu.integrate(raw, K640, w2c)
        ko.integrate(ref, raw, K640, w2c, ko.integration_options(mode=abi.KF_INTEGRATION_BAND),
                     abi.KF_RULE_ANGLE_WEIGHTED)
    assert np.array_equal(gpu.block_grid() != 0xFFFFFFFF, ref.grid != 0xFFFFFFFF)
    o = ko.raycast_options(corner_policy=policy, step_scale=scale, cell_gradient_normals=cell_normals)
    half = 0.5 * res[0] * vs
    hits = 0
    # widths of the three lane counts per ray (8, 2 and 1), odd extents; inside, beside and before the domain
    for width, height, pose in ((131, 97, turned(0.0, 0.2)), (251, 189, turned(0.1, -0.5, half + 0.3)),
                                (401, 303, turned(1.4, 0.1)), (131, 97, turned(0.5, 0.0)), (251, 189, turned(0.0, 0.0))):
        k = abi.Intrinsics(0.8 * width, 0.8 * width, 0.5 * width, 0.5 * height)
        maps = gpu.raycast(k, width, height, pose)
        p, n, c = ko.raycast(ref, k, width, height, pose, o, threads=8)
        assert same(maps.points, p) and same(maps.normals, n) and same(maps.colors, c), (width, pose[:3, 3])
        hits += int(np.isfinite(p).all(-1).sum())
    assert hits > 0 or max(res) < 16
