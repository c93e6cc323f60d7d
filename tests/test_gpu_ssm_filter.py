"""The matrix builder's FP32 filter against the oracle's ray-driven builder where
its margins are tightest: voxels much smaller and much larger than a channel, a
grid of odd size, two and many detector rows, each flying focal spot. Every
column's indices and FP32 weights equal the oracle's bit for bit."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
import oracle_util as O
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    # nch, rows, row_iso, views, phi, z, nx, fov, slice
    "fine": (64, 5, 0.06, 48, 0, 0, 21, 0.8, 0.06),
    "coarse": (96, 3, 0.9, 40, 0, 0, 6, 30.0, 1.7),
    "two rows": (48, 2, 1.5, 64, 0, 0, 9, 20.0, 1.5),
    "phi": (120, 12, 0.2, 40, 1, 0, 15, 11.0, 0.13),
    "z": (80, 8, 0.4, 40, 0, 1, 11, 9.0, 0.4),
    "phi z": (80, 8, 0.4, 32, 1, 1, 10, 12.0, 0.3),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_filtered_build_equals_oracle(ctx, tmp_path, name):
    nch, rows, row_iso, views, phi, z, nx, fov, thick = CASES[name]
    fan = 2.0 * np.arcsin(0.5 * max(fov, 4.0) / W.R_SRC) * 1.1 / nch
    prm = {**W._BASE, **W._scanner(nch, nch / 2.0 - 0.25, float(fan), rows, row_iso, views, bool(phi), 1.0, 6),
           **W._recon(nx, fov, thick, 2, -2.2 * rows * row_iso, "quadratic", 1.0, 0.005, 1)}
    if z:
        prm.update(Zffs=1, center_row=(rows / 2 - 1) / 2.0, Readings=6 * views * 2 * (2 if phi else 1))
    d = str(tmp_path)
    prm.update(sinogram_path=d + "/raw.bin", output_dir=d, output_file="o.img")
    open(d + "/raw.bin", "wb").close()
    rp = C.configure_recon_params(W.write_prm(d + "/c.prm", prm))
    C.slice_tables(rp, allow_bad_range=True)  # sets table_direction
    ref = O.port_ssm(rp)
    assert ref.nnz > 0
    ssm = C.Ssm.generate(rp, ctx, C.SSM_FP32)
    assert ssm.info().nnz == ref.nnz
    for c in range(nx * nx):
        idx, w = ssm.column(c)
        ri, rw = ref.column(c)
        assert np.array_equal(idx, ri) and np.array_equal(w.view(np.int32), rw.view(np.int32)), (name, c)
