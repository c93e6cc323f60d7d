"""Grouped ICD launches: one reconstruction moved between matrices, and the
update kernel at the edges of its dispatch."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_recon_follows_a_replaced_matrix(ctx, tmp_path):
    """A matrix freed and built again may come back at the same addresses:
    what a reconstruction captured or counted for the first must not serve
    the second. One update in flight, so the iterates are reproducible."""
    _, rp = W.materialise("small", str(tmp_path))
    data = C.load_raw(rp)
    opts = C.icd_opts(mode=C.ICD_GROUPED, weights=C.SSM_FP16, warps_in_flight=1)
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
