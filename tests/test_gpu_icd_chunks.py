"""The one-warp ICD kernels at the remainders of their chunks (256 and 512 entries):
a scan whose field of view holds a single voxel, so that an iteration is one
update, over columns from shorter than a chunk to many chunks and a remainder.
Each must give the step of the eight-warp kernel, which sums in another order:
FP32 partial sums of n terms differ by a few n^(1/2) 2^-24 of their absolute sum,
under 1e-5 of the step here."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views,ffs", [(9, False), (23, True), (64, False), (101, True), (257, False)])
def test_single_update_over_chunk_remainders(ctx, tmp_path, views, ffs):
    d = str(tmp_path)
    prm = {**W._BASE, **W._scanner(48, 23.75, 0.00882, 4, 1.5, views, ffs, 1.0, 5),
           **W._recon(5, 25.0, 1.5, 1, -7.0, "quadratic", 5.0, 0.005, 1),
           "acquisition_fov": 2.0, "sinogram_path": d + "/raw.bin", "output_dir": d, "output_file": "o.img"}
    open(d + "/raw.bin", "wb").close()
    rp = C.configure_recon_params(W.write_prm(d + "/c.prm", prm))
    tables = C.slice_tables(rp)
    raw = np.random.default_rng(views).uniform(0.5, 3.0, rp.raw_shape).astype(np.float32)
    ssm = C.Ssm.generate(rp, ctx, C.SSM_BOTH)

    def one(**o):
        rc = C.Recon(rp, tables.slice_indices, ctx)
        rc.set_raw(raw)
        rc.set_volume(ssm, None)
        st = rc.iterate(ssm, 1, C.icd_opts(mode=C.ICD_GROUPED, **o))
        rc.refresh_residual(ssm)
        v, cost = rc.volume(), rc.cost()
        rc.free()
        assert np.count_nonzero(v) == 1, "one voxel inside the field of view"
        return float(v.max()), st.entries, cost

    for weights in (C.SSM_FP32, C.SSM_FP16):
        ref, n, cost = one(weights=weights, warps_per_voxel=8, warps_in_flight=8, entry_pairs=-1)
        assert n > 0
        for epl in (8, 16):
            for pairs in (0, -1) if weights == C.SSM_FP16 else (0,):
                got, m, c = one(weights=weights, entries_per_lane=epl, entry_pairs=pairs)
                assert m == n
                assert abs(got - ref) <= 1e-5 * abs(ref), (epl, pairs, got, ref)
                assert abs(c - cost) <= 1e-5 * abs(cost)
