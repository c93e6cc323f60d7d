"""What the ICD kernels write into the error sinogram, at the remainders of their chunks
(256 and 512 entries, 1024 pairs): a scan whose field of view holds a single voxel and whose
raw data are that voxel's rays times x0, so that one update with a vanishing penalty leaves
e = 0 and the cost over e shows each entry that the reductions missed, doubled or misplaced.

Of n entries a_i, each is left with x0 a_i times the rounding of du (alpha and beta are sums
of n FP32 terms, n^(1/2) 2^-24 of them at most a few times over: under 1e-5 for n of 10^5),
of its raw value and of one FP32 product and sum: together under 2e-5 x0 a_i. The cost is
0.5 sum e^2 and stays under 0.5 (2e-5)^2 x0^2 sum a_i^2; one entry of a hundredth of the
largest's weight left out shows as long as (a_max / 100)^2 is above 4e-10 sum a_i^2."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu
X0 = 0.75


@pytest.mark.parametrize("views,ffs", [(9, False), (23, True), (64, False), (101, True), (257, False), (700, True)])
@pytest.mark.parametrize("weights", [C.SSM_FP32, C.SSM_FP16])
def test_single_update_empties_the_error(ctx, tmp_path, views, ffs, weights):
    d = str(tmp_path)
    prm = {**W._BASE, **W._scanner(47, 23.75, 0.00882, 5, 1.5, views, ffs, 1.0, 5),
           **W._recon(5, 25.0, 1.5, 1, -10.0, "quadratic", 1e-12, 0.005, 1),
           "acquisition_fov": 2.0, "sinogram_path": d + "/raw.bin", "output_dir": d, "output_file": "o.img"}
    open(d + "/raw.bin", "wb").close()
    rp = C.configure_recon_params(W.write_prm(d + "/c.prm", prm))
    tables = C.slice_tables(rp)
    ssm = C.Ssm.generate(rp, ctx, weights)
    # the column's rays (FP16 weights as stored), at the slice's views
    idx, w = ssm.column(2 + 5 * 2)
    q = idx.astype(np.int64) + (int(tables.slice_indices[0]) - int(rp.geom.num_views_for_system_matrix) // 2) * 47 * 5
    raw = np.zeros(int(np.prod(rp.raw_shape)), np.float32)
    seen = (q >= 0) & (q < raw.size)
    raw[q[seen]] = np.float32(X0) * w[seen]
    assert seen.sum() > 0
    bound = 0.5 * (2e-5 * X0) ** 2 * float((w[seen].astype(np.float64) ** 2).sum())
    missed = 0.5 * (X0 * 0.01 * float(w.max())) ** 2
    assert missed > bound

    one_warp = [dict(entries_per_lane=e, entry_pairs=p) for e in (8, 16)
                for p in ((0, -1) if weights == C.SSM_FP16 else (0,))]
    many = [dict(warps_per_voxel=v, entry_pairs=-1) for v in (4, 8)]
    staged = [dict(stage_column=s) for s in (1, 2, 3)]
    if weights == C.SSM_FP16:
        many += [dict(warps_per_voxel=v) for v in (4, 8)]
        staged += [dict(stage_column=s, warps_per_voxel=8) for s in (4, 5, 6)]
    for more in one_warp + many + staged:
        rc = C.Recon(rp, tables.slice_indices, ctx)
        rc.set_raw(raw.reshape(rp.raw_shape))
        rc.set_volume(ssm, None)
        st = rc.iterate(ssm, 1, C.icd_opts(weights=weights, **more))
        assert st.entries == seen.sum(), more
        v, cost = rc.volume(), rc.cost()
        rc.free()
        assert np.count_nonzero(v) == 1 and abs(float(v.max()) - X0) <= 1e-5 * X0, (more, v.max())
        assert cost <= bound, (more, cost, bound)
    ssm.free()
