"""A reset writes only the bricks that integrations wrote, and the observed
count reads only those: after any use the storage equals a new volume's, bit
for bit, and the count is the number of voxels with a weight."""

import numpy as np
import pytest

import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.fixture(scope="module")
def seq():
    return synthetic.make_sequence(seed=31, frames=2, max_step_m=0.2, max_step_deg=20.0)


def make(res, voxel, color, sparse, capacity=0):
    vs = 5.12 / max(res)
    return kf.Pipeline(kf.pipeline_config(
        res, vs, (-0.5 * res[0] * vs, -0.5 * res[1] * vs, -0.5), max(0.05, 3 * vs), voxel=voxel,
        color=abi.KF_COLOR_FLOAT if color else abi.KF_COLOR_NONE, sparse_block_capacity=capacity,
        storage=abi.KF_STORAGE_SPARSE if sparse else abi.KF_STORAGE_DENSE,
        integration_mode=abi.KF_INTEGRATION_BAND if sparse else abi.KF_INTEGRATION_FULL))


def storage(gpu, color, sparse):
    raw = (gpu.download_pool() if sparse else gpu.download_raw()).view(np.uint32)
    return (raw,) + ((gpu.host_view(with_color=True)[2],) if color else ())


@pytest.mark.parametrize("res,voxel,color,sparse,capacity", [
    ((71, 53, 64), abi.KF_VOXEL_FLOAT, True, False, 0),
    ((7, 8, 9), abi.KF_VOXEL_QUANTIZED, False, False, 0),
    ((130, 129, 127), abi.KF_VOXEL_BF16, True, False, 0),
    ((96, 96, 96), abi.KF_VOXEL_FLOAT, True, True, 0),
    ((96, 96, 96), abi.KF_VOXEL_QUANTIZED, False, True, 100),  # the pool overflows
])
def test_reset_equals_a_new_volume(seq, res, voxel, color, sparse, capacity):
    gpu, fresh = make(res, voxel, color, sparse, capacity), make(res, voxel, color, sparse, capacity)
    empty = storage(fresh, color, sparse)
    assert gpu.observed_voxel_count() == 0
    gpu.reset()  # before any use
    for f in range(2):
        gpu.integrate(seq.depth[f], K640, np.linalg.inv(seq.poses[f]), color=seq.color[f] if color else None)
    used = storage(gpu, color, sparse)
    assert any(not np.array_equal(a, b) for a, b in zip(used, empty))
    weight = used[0][..., 1].view(np.float32) if voxel == abi.KF_VOXEL_FLOAT else used[0] >> 16
    assert gpu.observed_voxel_count() == int((weight > 0).sum())
    gpu.reset()
    assert all(np.array_equal(a, b) for a, b in zip(storage(gpu, color, sparse), empty))
    assert gpu.observed_voxel_count() == 0
    # and the next sequence starts from it
    gpu.integrate(seq.depth[0], K640, np.linalg.inv(seq.poses[0]), color=seq.color[0] if color else None)
    fresh.integrate(seq.depth[0], K640, np.linalg.inv(seq.poses[0]), color=seq.color[0] if color else None)
    assert all(np.array_equal(a, b) for a, b in zip(storage(gpu, color, sparse), storage(fresh, color, sparse)))
