"""The matrix builder's FP32 filter on grids away from the isocentre: slices above and below
the source's plane, fields of view beside the axis, one detector row. Count and fill must
agree (the build refuses otherwise) and every column equal the oracle's ray-driven builder
bit for bit."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
import oracle_util as O
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    # rows, row_iso, phi, z, slice, voxels off the isocentre in x, y, z
    "above": (8, 0.4, 0, 0, 0.2, 0.0, 0.0, 4.0),
    "far below, thin slices": (12, 0.3, 1, 0, 0.045, 0.0, 0.0, -15.5),
    "beside": (6, 0.5, 1, 0, 0.3, 7.25, -11.0, 0.0),
    "all": (8, 0.4, 1, 1, 0.3, -6.5, 9.0, 5.5),
    "one row": (1, 2.0, 0, 0, 1.0, 0.0, 0.0, 0.0),
    "outside": (4, 0.3, 0, 0, 0.3, 0.0, 0.0, 40.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_build_off_centre_equals_oracle(ctx, tmp_path, name):
    rows, row_iso, phi, z, thick, ox, oy, oz = CASES[name]
    nch, views, nx, fov = 96, 40, 12, 6.0
    fan = 2.0 * np.arcsin(0.5 * 20.0 / W.R_SRC) * 1.1 / nch
    prm = {**W._BASE, **W._scanner(nch, nch / 2.0 - 0.25, float(fan), rows, row_iso, views, bool(phi), 1.0, 8),
           **W._recon(nx, fov, thick, 2, -2.2 * rows * row_iso, "quadratic", 1.0, 0.005, 1)}
    prm["center_row"] = max(prm["center_row"], 0.1)
    if z:
        prm.update(Zffs=1, center_row=(rows / 2 - 1) / 2.0, Readings=8 * views * 2 * (2 if phi else 1))
    d = str(tmp_path)
    prm.update(sinogram_path=d + "/raw.bin", output_dir=d, output_file="o.img")
    open(d + "/raw.bin", "wb").close()
    rp = C.configure_recon_params(W.write_prm(d + "/c.prm", prm))
    C.slice_tables(rp, allow_bad_range=True)  # sets table_direction
    rp.geom.center_voxel_x += ox
    rp.geom.center_voxel_y += oy
    rp.geom.center_voxel_z += oz
    ref = O.port_ssm(rp)
    ssm = C.Ssm.generate(rp, ctx, C.SSM_FP32)
    assert ssm.info().nnz == ref.nnz and (ref.nnz == 0) == (name == "outside")
    for c in range(nx * nx):
        idx, w = ssm.column(c)
        ri, rw = ref.column(c)
        assert np.array_equal(idx, ri) and np.array_equal(w.view(np.int32), rw.view(np.int32)), (name, c)
