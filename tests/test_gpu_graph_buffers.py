"""A recorded frame graph is used only on the buffers it was recorded on: other
calls between two frames may replace them (a frame integrated or a pyramid built
at another size) or change what its kernels were given (other intrinsics, another
pyramid or tracker at an address that was free).  The frames equal, bit for bit,
those of a loop without such calls."""

import ctypes as C
import gc

import numpy as np
import pytest

import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)
FRAMES = 5


@pytest.fixture(scope="module")
def seq():
    return synthetic.make_sequence(seed=91, frames=FRAMES)


def run(seq, between=None, renew=False, intrinsics=lambda f: K640):
    half = 0.5 * 128 * 0.02
    gpu = kf.Pipeline(kf.pipeline_config(128, 0.02, (-half, -half, -0.5), 0.05, color=abi.KF_COLOR_NONE))
    lib, iterations = abi.load(), (C.c_uint32 * 4)(*kf.ICP_ITERATIONS)
    pyramid, tracker = kf.PyramidSource(), kf.ProjectiveIcpTracker()
    pose, out = abi.rigid_from_matrix(seq.poses[0]), []
    for f in range(FRAMES):
        if f and between is not None:
            between(gpu, pyramid, f)
        if f and renew:
            pyramid = tracker = None
            gc.collect()
            pyramid, tracker = kf.PyramidSource(), kf.ProjectiveIcpTracker()
        depth, result = np.ascontiguousarray(seq.depth[f]), abi.FrameResult()
        abi.check(lib.kf_frame_process(gpu.handle, pyramid.handle, tracker.handle, depth.ctypes.data_as(C.c_void_p),
                                       None, 640, 480, intrinsics(f), abi.KF_MEMORY_HOST, iterations, 1 if f == 0 else 0,
                                       C.byref(pose), C.byref(result)))
        out.append((result.tracked, np.array(abi.matrix_from_rigid(pose))))
    return out, gpu.download_raw().view(np.uint32)


def same(a, b):
    return all(x[0] == y[0] and np.array_equal(x[1], y[1]) for x, y in zip(a[0], b[0])) and np.array_equal(a[1], b[1])


@pytest.fixture(scope="module")
def plain(seq):
    out = run(seq)
    assert all(tracked for tracked, _ in out[0])
    return out


def small(k):
    return abi.Intrinsics(k.fx / 2, k.fy / 2, k.cx / 2, k.cy / 2)


def test_a_frame_integrated_at_another_size(seq, plain):
    def between(gpu, pyramid, f):  # without a usable depth: it changes nothing in the volume
        shape = (240, 320) if f % 2 else (700, 900)
        gpu.integrate(np.zeros(shape, dtype=np.uint16), small(K640), np.eye(4))
    assert same(run(seq, between), plain)


def test_a_pyramid_built_at_another_size(seq, plain):
    def between(gpu, pyramid, f):
        pyramid.build(np.full((240, 320), 5000, dtype=np.uint16), small(K640))
        if f % 2:
            pyramid.build(np.full((480, 640), 5000, dtype=np.uint16), K640)  # and back: the size is the frames' again
    assert same(run(seq, between), plain)


def test_new_pyramids_and_trackers(seq, plain):
    assert same(run(seq, renew=True), plain)


def test_intrinsics_that_a_build_already_brought(seq):
    other = abi.Intrinsics(K640.fx * 1.01, K640.fy * 1.01, K640.cx, K640.cy)

    def which(f):
        return other if f >= 2 else K640

    def between(gpu, pyramid, f):
        pyramid.build(seq.depth[0], which(f))
    assert same(run(seq, between, intrinsics=which), run(seq, renew=True, intrinsics=which))
