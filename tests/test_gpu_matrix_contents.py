"""One reconstruction given one matrix after another, each of other contents: a geometry that
a reconstruction accepts may have another fan increment, centre channel or voxel size. What
was captured or counted for one matrix must not serve the next, wherever it is allocated."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _change(geom, k):
    if k == 1:
        geom.center_channel_non_ffs += 1.5
    elif k == 2:
        geom.voxel_size_x *= 0.8
        geom.voxel_size_y *= 0.8
    elif k == 3:
        geom.fan_angle_increment *= 1.15
        geom.transaxial_detector_spacing *= 1.15


@pytest.mark.parametrize("stage", [0, 4])
def test_each_matrix_is_used(ctx, tmp_path, stage):
    """Eight updates in flight: two runs with one matrix differ by under 1e-3 in the image
    (their order), the matrices' images and entry counts by far more."""
    _, rp = W.materialise("small", str(tmp_path))
    data = C.load_raw(rp)
    opts = C.icd_opts(weights=C.SSM_FP16, warps_per_voxel=8, warps_in_flight=8, stage_column=stage)
    original = {f: getattr(rp.geom, f) for f in ("center_channel_non_ffs", "voxel_size_x", "voxel_size_y",
                                                 "fan_angle_increment", "transaxial_detector_spacing")}

    def matrix(k):
        for f, v in original.items():
            setattr(rp.geom, f, v)
        _change(rp.geom, k)
        ssm = C.Ssm.generate(rp, ctx, C.SSM_BOTH)
        for f, v in original.items():
            setattr(rp.geom, f, v)
        return ssm

    def once(rc, ssm):
        rc.set_volume(ssm, None)
        st = rc.iterate(ssm, 1, opts)
        return rc.volume().astype(np.float64), st.entries

    want = []
    for k in range(4):
        rc, ssm = C.Recon(rp, data.slice_indices, ctx), matrix(k)
        rc.set_raw(data.raw)
        want.append(once(rc, ssm))
        rc.free()
        ssm.free()
    for i in range(4):
        for j in range(i):
            assert want[i][1] != want[j][1]
            assert np.linalg.norm(want[i][0] - want[j][0]) > 0.02 * np.linalg.norm(want[j][0])
    rc = C.Recon(rp, data.slice_indices, ctx)
    rc.set_raw(data.raw)
    for k in (0, 1, 2, 3, 1, 0, 3):  # each freed before the next is built
        ssm = matrix(k)
        v, n = once(rc, ssm)
        assert n == want[k][1], k
        assert np.linalg.norm(v - want[k][0]) <= 1e-3 * np.linalg.norm(want[k][0]), k
        ssm.free()
    held = [matrix(k) for k in range(4)]  # and all held at once
    for k in (2, 0, 3, 1, 2):
        v, n = once(rc, held[k])
        assert n == want[k][1] and np.linalg.norm(v - want[k][0]) <= 1e-3 * np.linalg.norm(want[k][0]), k
    rc.free()
