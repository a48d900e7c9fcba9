"""A pipeline keeps at most 256 MB of device memory of its meshes' working
arrays, both of them together: a rough surface of some 1.5 million vertices
needs more, though neither array does, and one is given back; the mesh of the
next call, on a new array, is the same.  That mesh is larger than the
page-locked staging too, so it comes back by direct copies; a smaller one of the
same volume goes through the staging, and is the part of the large one's
vertices that its threshold keeps."""

import numpy as np
import pytest

import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)
MB = 1 << 20


def test_kept_memory_is_bounded():
    import torch  # memory counters only
    rng = np.random.default_rng(5)
    pipeline = kf.Pipeline(kf.pipeline_config(384, 0.01, (-1.92, -1.92, 0.3), 0.6, color=abi.KF_COLOR_NONE))
    for f in range(2):
        depth = (5000 * (2.2 + 0.5 * rng.standard_normal((480, 640)))).clip(0, 20000).astype(np.uint16)
        depth[:, :210], depth[:, 430 if f == 0 else 240:] = 0, 0  # a strip, and a part of it seen twice
        pipeline.integrate(depth, K640, np.eye(4))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    first = pipeline.extract_mesh()
    kept = free - torch.cuda.mem_get_info()[0]
    vertices, corners = len(first["positions"]), 3 * len(first["triangles"])
    # what the two arrays of the call hold: per vertex 136 bytes, per corner 8
    cells = 384 ** 3 * 3 // 32 * 4 * 2  # bits and ranks of the volume's edges
    surface = 136 * vertices + 8 * corners
    assert surface < 256 * MB < cells + surface
    assert 36 * vertices + 4 * corners > 64 * MB
    assert kept <= 256 * MB + 8 * MB  # allocation granularity
    again, small = pipeline.extract_mesh(), pipeline.extract_mesh(1.5)
    for name in first:
        assert np.array_equal(first[name], again[name], equal_nan=first[name].dtype.kind == "f"), name
    assert 0 < 36 * len(small["positions"]) + 12 * len(small["triangles"]) < 64 * MB
    rows = {tuple(v) for v in first["positions"]}
    assert all(tuple(v) in rows for v in small["positions"])
