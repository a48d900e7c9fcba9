"""The whole-level ICP kernel keeps its live maps in shared memory between the
sweeps of a level (up to 1.2 million live pixels; larger images re-read them)
and computes the diagnostics' eigenvalues once, after the last step:

* the second step's sums equal, bit for bit, one sweep from the maps at the
  pose the first step reached, below and above that size and at odd sizes;
* the eigenvalue diagnostics are those of the last step's normal equations."""

import ctypes as C

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

RES, VOXEL, ORIGIN, TRUNC = 128, 0.04, (-2.56, -2.56, -0.5), 0.12


def device(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(scope="module")
def scene():
    seq = synthetic.make_sequence(seed=21, frames=2)
    k = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)
    gpu = kf.Pipeline(kf.pipeline_config(RES, VOXEL, ORIGIN, TRUNC, color=abi.KF_COLOR_NONE))
    normals = ko.pyramid(seq.depth[0], k, ko.depth_options())[0]["normals"]
    gpu.integrate(seq.depth[0], k, ko.rigid_inverse(abi.rigid_from_matrix(seq.poses[0])), normals=normals)
    return gpu, seq


# 37x29: one CTA; 640x480: 4 or 5 pixels a thread; 1280x947 and 1300x960: 16
# and 17, the last size kept and the first one not
@pytest.mark.parametrize("width,height", [(37, 29), (640, 480), (1280, 947), (1300, 960)])
def test_second_step_equals_a_sweep_from_the_maps(scene, width, height):
    gpu, seq = scene
    lib = abi.load()
    scale = max(width / 640, height / 480)
    rows = np.minimum((np.arange(height) / scale).astype(int), 479)
    cols = np.minimum((np.arange(width) / scale).astype(int), 639)
    depth = seq.depth[1][np.ix_(rows, cols)]
    k = abi.Intrinsics(synthetic.FX * scale, synthetic.FY * scale, synthetic.CX * scale, synthetic.CY * scale)
    pyr = kf.PyramidSource()
    pyr.build(depth, k)
    live = pyr.level(0)
    maps = gpu.raycast(k, width, height, seq.poses[0])
    points, normals = device(maps.points), device(maps.normals)
    tracker = kf.ProjectiveIcpTracker()
    start = abi.rigid_from_matrix(seq.poses[0])
    model = ko.rigid_inverse(start)
    p, n = C.c_void_p(points.data_ptr()), C.c_void_p(normals.data_ptr())

    def level(steps):
        out, sums = abi.IcpOutcome(), np.empty(29, dtype=np.float32)
        abi.check(lib.kf_icp_level(tracker.handle, C.byref(live), p, n, width, height, k, C.byref(model),
                                   C.byref(start), steps, C.byref(out), sums.ctypes.data_as(C.c_void_p)))
        return out, sums

    first, _ = level(1)
    assert first.iterations == 1 and first.status == abi.KF_ICP_MAX_ITERATIONS
    second, sums = level(2)
    assert second.iterations == 2
    expected, count = np.empty(29, dtype=np.float32), C.c_uint64()
    abi.check(lib.kf_icp_normal_equations(tracker.handle, C.byref(live), p, n, width, height, k,
                                          C.byref(first.pose), C.byref(model),
                                          expected.ctypes.data_as(C.c_void_p), C.byref(count)))
    assert np.array_equal(sums.view(np.uint32), expected.view(np.uint32))
    assert second.correspondences == count.value > 64
    # FP64 eigenvalues of the FP32 sums, rounded once to float
    a = np.zeros((6, 6))
    a[np.triu_indices(6)] = sums[:21]
    eig = np.linalg.eigvalsh(a + np.triu(a, 1).T)
    assert np.isclose(second.min_system_eigenvalue, eig[0], rtol=1e-6)
    assert np.isclose(second.condition_number, eig[-1] / eig[0], rtol=1e-6)
