"""One reconstruction moved between matrices, and one matrix between scans."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_recon_follows_a_replaced_matrix(ctx, tmp_path):
    """A matrix freed and built again may come back at the same addresses:
    what a reconstruction captured or counted for the first must not serve
    the second. One update in flight (one CTA of 8 warps; the one-warp kernels round
    up to 8 updates), so the iterates are reproducible."""
    _, rp = W.materialise("small", str(tmp_path))
    data = C.load_raw(rp)
    opts = C.icd_opts(mode=C.ICD_GROUPED, weights=C.SSM_FP16, warps_per_voxel=8, warps_in_flight=8)
    out = []
    rc = C.Recon(rp, data.slice_indices, ctx)
    rc.set_raw(data.raw)
    for _ in range(3):
        ssm = C.Ssm.generate(rp, ctx, C.SSM_BOTH)
        rc.set_volume(ssm, None)
        st = rc.iterate(ssm, 1, opts)
        out.append((rc.volume(), st.entries))
        ssm.free()
    rc.free()
    for v, n in out[1:]:
        # FP32 partial sums are ordered alike; only the reductions into e race
        assert np.linalg.norm(v - out[0][0]) <= 1e-5 * np.linalg.norm(out[0][0])
        assert n == out[0][1] > 0


@pytest.mark.parametrize("mode", [C.ICD_SEQUENTIAL, C.ICD_GROUPED])
@pytest.mark.parametrize("longer_first", [False, True])
def test_matrix_shared_by_scans_of_different_length(ctx, tmp_path, mode, longer_first):
    """The matrix does not depend on the number of views of a scan: one built for
    a shorter or longer scan gives the iterates of the scan's own. The same
    slices and raw data of the common views; one update in flight."""
    _, rp = W.materialise("small", str(tmp_path / "a"))
    data = C.load_raw(rp)
    n = int(rp.geom.Readings)
    _, rp2 = W.materialise("small", str(tmp_path / "b"), raw=False, overrides=dict(Readings=n + 197))
    raw2 = np.zeros(rp2.raw_shape, np.float32)
    raw2[:n] = data.raw
    scans = [(rp, data.raw), (rp2, raw2)]
    opts = C.icd_opts(mode=mode, weights=C.SSM_FP32 if mode == C.ICD_SEQUENTIAL else C.SSM_FP16, warps_per_voxel=8,
                      warps_in_flight=8, compute_cost=True)

    def run(i, ssm):
        r, raw = scans[i]
        rc = C.Recon(r, data.slice_indices, ctx)
        rc.set_raw(raw)
        rc.set_volume(ssm, None)
        cost = rc.iterate(ssm, 2, opts).cost
        rc.refresh_residual(ssm)
        out = rc.volume_f64(), cost
        rc.free()
        return out

    rp2.geom.table_direction = rp.geom.table_direction
    own = [run(i, C.Ssm.generate(scans[i][0], ctx, C.SSM_BOTH)) for i in (0, 1)]
    ssm = C.Ssm.generate(rp, ctx, C.SSM_BOTH)
    for i in ((1, 0, 1) if longer_first else (0, 1, 0)):
        v, cost = run(i, ssm)
        assert np.linalg.norm(v - own[i][0]) <= 1e-5 * np.linalg.norm(own[i][0])
        assert abs(cost - own[i][1]) <= 1e-5 * own[i][1]


def test_autotune_refuses_a_matrix_of_another_geometry(ctx, tmp_path):
    """The refusal comes before the matrix and the scan settle on one layout."""
    _, rp = W.materialise("small", str(tmp_path / "a"))
    _, other = W.materialise("tiny", str(tmp_path / "b"))
    data = C.load_raw(rp)
    rc = C.Recon(rp, data.slice_indices, ctx)
    rc.set_raw(data.raw)
    ssm = C.Ssm.generate(rp, ctx, C.SSM_BOTH)
    ssm_other = C.Ssm.generate(other, ctx, C.SSM_BOTH)
    rc.set_volume(ssm, None)
    mid = int(ssm_other.info().n_columns) // 2
    before = ssm_other.column(mid)
    with pytest.raises(C.CtbbError, match="geometry does not match"):
        rc.autotune(ssm_other, C.icd_opts(mode=C.ICD_GROUPED, weights=C.SSM_FP16))
    after = ssm_other.column(mid)
    assert all(np.array_equal(a, b) for a, b in zip(before, after))
    for o in (rc, ssm, ssm_other):
        o.free()
