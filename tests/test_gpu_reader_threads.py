"""Several threads count and mesh one pipeline at once: the calls share the
pipeline's working memory and take turns, so every one of them returns what a
single call returns.  The two mesh thresholds need arrays of different sizes,
so calls that overlapped would resize them under one another."""

import concurrent.futures

import numpy as np
import pytest

import kf_oracle as ko
import kinectfusion_b200 as kf
from kinectfusion_b200 import abi, synthetic

pytestmark = pytest.mark.gpu

K640 = abi.Intrinsics(synthetic.FX, synthetic.FY, synthetic.CX, synthetic.CY)


@pytest.mark.parametrize("sparse", [False, True])
def test_counts_and_meshes_from_several_threads(sparse):
    seq = synthetic.make_sequence(seed=71, frames=3, max_step_m=0.1, max_step_deg=8.0)
    pipeline = kf.Pipeline(kf.pipeline_config(
        160, 0.032, (-2.56, -2.56, -0.5), 0.1, color=abi.KF_COLOR_NONE,
        storage=abi.KF_STORAGE_SPARSE if sparse else abi.KF_STORAGE_DENSE,
        integration_mode=abi.KF_INTEGRATION_BAND if sparse else abi.KF_INTEGRATION_FULL))
    for f in range(3):
        pipeline.integrate(seq.depth[f], K640, ko.rigid_inverse(abi.rigid_from_matrix(seq.poses[f])))
    # an observation without normals weighs 1: the second threshold needs two of them
    weights = (0.0, 1.5)
    count, meshes = pipeline.observed_voxel_count(), {w: pipeline.extract_mesh(w) for w in weights}
    sizes = [meshes[w]["triangles"].shape[0] for w in weights]
    assert count > 0 and sizes[0] > sizes[1] > 0

    def work(i):
        bad = 0
        for r in range(12):
            if (i + r) % 3 == 0:
                bad += pipeline.observed_voxel_count() != count
            else:
                w = weights[(i + r) % 2]
                got = pipeline.extract_mesh(w)
                bad += not all(np.array_equal(got[name], meshes[w][name]) for name in got)
        return bad

    with concurrent.futures.ThreadPoolExecutor(6) as pool:
        assert sum(pool.map(work, range(6))) == 0
