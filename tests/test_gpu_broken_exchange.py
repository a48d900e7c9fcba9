"""Frames behind an ICP exchange that gave up (kf_tracker_stall_next_level makes
one on purpose; its waits are bounded, nothing hangs).

Until the host has read a result that shows it, no frame is tracked or fused,
the ones already queued included; reading it restarts the exchange from the
device's own step count, so neither the packets left behind nor a late read of
an older result can reach a later step.  The frames after it are, bit for bit,
those of a tracker that never stalled."""

import ctypes as C

import numpy as np
import pytest

import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.fixture(scope="module")
def seq():
    return synthetic.make_sequence(seed=61, frames=4)


class Loop:
    def __init__(self, seq):
        half = 0.5 * 128 * 0.02
        self.pipeline = kf.Pipeline(kf.pipeline_config(128, 0.02, (-half, -half, -0.5), 0.05, color=abi.KF_COLOR_NONE))
        self.pyramid, self.tracker = kf.PyramidSource(), kf.ProjectiveIcpTracker()
        self.depth = [np.ascontiguousarray(d) for d in seq.depth]
        self.iterations = (C.c_uint32 * 4)(*kf.ICP_ITERATIONS)
        self.lib = abi.load()

    def _send(self, call, f):
        abi.check(call(self.pipeline.handle, self.pyramid.handle, self.tracker.handle,
                       self.depth[f].ctypes.data_as(C.c_void_p), None, 640, 480, K640, abi.KF_MEMORY_HOST,
                       self.iterations, 1 if f == 0 else 0))

    def enqueue(self, f):
        self._send(self.lib.kf_frame_enqueue, f)

    def submit(self, f):
        self._send(self.lib.kf_frame_submit, f)

    def _read(self, call):
        result = abi.FrameResult()
        return call(self.pipeline.handle, C.byref(result)), result

    def fetch(self):
        return self._read(self.lib.kf_frame_result_fetch)

    def next(self):
        return self._read(self.lib.kf_frame_result_next)

    def stall(self):
        abi.check(self.lib.kf_tracker_stall_next_level(self.tracker.handle))

    def updates(self):
        n = C.c_uint64()
        abi.check(self.lib.kf_pipeline_update_counts(self.pipeline.handle, C.byref(n), None))
        return n.value


def pose(status, result):
    assert status == abi.KF_OK and result.tracked
    return np.array(abi.matrix_from_rigid(result.camera_to_world))


@pytest.fixture(scope="module")
def clean(seq):
    """Poses after each frame and the volume after frames 2 and 3 of a loop that never stalled."""
    loop, poses, volumes = Loop(seq), [], []
    for f in range(4):
        loop.enqueue(f)
        poses.append(pose(*loop.fetch()))
        volumes.append(loop.pipeline.download_raw().view(np.uint32))
    return poses, volumes


def start(seq, clean):
    loop = Loop(seq)
    for f in range(2):
        loop.enqueue(f)
        assert np.array_equal(pose(*loop.fetch()), clean[0][f])
    loop.stall()
    return loop


def test_queued_frames_fail_and_the_next_one_is_clean(seq, clean):
    poses, volumes = clean
    loop = start(seq, clean)
    fused = loop.updates()
    loop.enqueue(2)
    loop.enqueue(3)  # queued behind the broken exchange
    assert loop.fetch()[0] == abi.KF_ERR_DEVICE_TIMEOUT
    assert loop.updates() == fused
    for f in (2, 3):
        loop.enqueue(f)
        assert np.array_equal(pose(*loop.fetch()), poses[f])
        assert np.array_equal(loop.pipeline.download_raw().view(np.uint32), volumes[f])


def test_a_late_read_moves_nothing_back(seq, clean):
    poses, volumes = clean
    loop = start(seq, clean)
    loop.submit(2)
    loop.submit(3)
    assert loop.next()[0] == abi.KF_ERR_DEVICE_TIMEOUT
    loop.enqueue(2)  # runs on the restarted exchange
    assert np.array_equal(pose(*loop.fetch()), poses[2])
    assert loop.next()[0] == abi.KF_ERR_DEVICE_TIMEOUT  # the older result, read late
    loop.enqueue(3)
    assert np.array_equal(pose(*loop.fetch()), poses[3])
    assert np.array_equal(loop.pipeline.download_raw().view(np.uint32), volumes[3])


def test_an_error_leaves_the_result_queue(seq, clean):
    poses, volumes = clean
    loop = start(seq, clean)
    fused = loop.updates()
    for f in (2, 3, 2, 3, 2, 3, 2, 3):
        loop.submit(f)  # eight results wait: the queue is full
    for _ in range(8):
        assert loop.next()[0] == abi.KF_ERR_DEVICE_TIMEOUT
    assert loop.next()[0] == abi.KF_ERR_INVALID_ARGUMENT  # nothing waits any more
    assert loop.updates() == fused
    loop.submit(2)
    loop.submit(3)
    for f in (2, 3):
        assert np.array_equal(pose(*loop.next()), poses[f])
    assert np.array_equal(loop.pipeline.download_raw().view(np.uint32), volumes[3])


def test_per_step_levels_fail_behind_a_broken_exchange_too(seq, clean):
    poses, volumes = clean
    loop = start(seq, clean)
    fused = loop.updates()
    loop.enqueue(2)
    loop.pipeline.set_concurrent(True)  # the levels as launches of their own, without an exchange
    loop.enqueue(3)
    assert loop.fetch()[0] == abi.KF_ERR_DEVICE_TIMEOUT
    assert loop.updates() == fused
    for f in (2, 3):
        loop.enqueue(f)
        assert np.array_equal(pose(*loop.fetch()), poses[f])
    assert np.array_equal(loop.pipeline.download_raw().view(np.uint32), volumes[3])
