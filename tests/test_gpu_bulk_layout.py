"""The bulk ICD kernels with more than three updates an SM in flight keep the error
sinogram and the entry pairs in a second layout (groups of two channels and two rows).
Detectors of odd and even size, matrices shared by scans of different length, and
changes between these kernels and the others.

What each check compares: the cost summed over the incrementally updated FP32 e against
that of y - A x recomputed in FP64 from the same image. An e of size s has been through k
additions of random rounding, an error of about s k^(1/2) 2^-24; with the data's s of 3 and
some thousand additions 1e-5, so the sums of squares of residuals near 1 agree to a few
1e-5. A wrong row, channel or view in any gather or reduction leaves another cost by more
than a part in a hundred."""
import numpy as np
import pytest

import ctbb_icd_b200 as C
from ctbb_icd_b200 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _scan(directory, nch, rows, ffs, extra=0):
    nx, nz, row_iso, views = 96, 40, 0.3, 60
    fan = 2.0 * np.arcsin(0.5 * 20.0 / W.R_SRC) / nch
    turns = int(np.ceil((nz * row_iso + 2.6 * rows * row_iso) / (rows * row_iso))) + (4 if rows > 1 else 8)
    prm = {**W._BASE, **W._scanner(nch, nch / 2.0 - 0.25, float(fan), rows, row_iso, views, ffs, 1.0, turns),
           **W._recon(nx, 18.0, row_iso, nz, (1.5 - 0.5 * turns) * rows * row_iso + 0.5 * nz * row_iso, "quadratic", 5.0,
                      0.005, 1), "sinogram_path": directory + "/raw.bin", "output_dir": directory, "output_file": "o.img"}
    prm["Readings"] += extra
    prm["center_row"] = max(prm["center_row"], 0.25)  # zero reads as missing
    open(directory + "/raw.bin", "wb").close()
    rp = C.configure_recon_params(W.write_prm(directory + "/c.prm", prm))
    return rp, C.slice_tables(rp)


class Scan:
    def __init__(self, ctx, directory, nch, rows, ffs, extra=0, tables=None):
        self.rp, own = _scan(directory, nch, rows, ffs, extra)
        self.tables = tables or own
        self.rc = C.Recon(self.rp, self.tables.slice_indices, ctx)
        self.exact = C.Recon(self.rp, self.tables.slice_indices, ctx)
        raw = np.random.default_rng(7).uniform(1.0, 3.0, self.rp.raw_shape).astype(np.float32)
        for r in (self.rc, self.exact):
            r.set_raw(raw)

    def check(self, ssm):
        self.exact.set_volume(ssm, self.rc.volume())
        want, got = self.exact.cost(), self.rc.cost()
        assert abs(got - want) <= TOL * want, (got, want)
        return want


def _opts(stage, warps=4736, **more):
    return C.icd_opts(weights=C.SSM_FP16, stage_column=stage, warps_per_voxel=8 if stage >= 4 else 1,
                      warps_in_flight=warps, lattice=16, **more)


@pytest.mark.parametrize("nch,rows,ffs", [(48, 4, False), (47, 5, False), (47, 4, True), (36, 3, False), (40, 2, False),
                                          (40, 1, False)])
@pytest.mark.parametrize("stage", [4, 5, 6])
def test_error_follows_the_image(ctx, tmp_path, nch, rows, ffs, stage):
    s = Scan(ctx, str(tmp_path), nch, rows, ffs)
    ssm = C.Ssm.generate(s.rp, ctx, C.SSM_BOTH)
    s.rc.set_volume(ssm, None)
    begin = s.rc.cost()
    if ssm.info().n_pairs == 0:  # built on first use; a single row's runs may not pair up
        try:
            s.rc.iterate(ssm, 1, _opts(stage))
        except C.CtbbError as e:
            assert rows == 1 and "entry pairs" in str(e)
            return
    s.rc.iterate(ssm, 2, _opts(stage))
    many = s.check(ssm)
    assert many < 0.9 * begin
    # the same iterations with the raw data's order (few updates in flight) descend alike
    s.rc.set_volume(ssm, None)
    s.rc.iterate(ssm, 3, _opts(stage, warps=1184))
    assert abs(s.check(ssm) - many) <= 0.05 * begin


@pytest.mark.parametrize("nch,rows", [(48, 4), (47, 5)])
def test_matrix_shared_by_scans_of_different_length(ctx, tmp_path, nch, rows):
    (tmp_path / "b").mkdir()
    a = Scan(ctx, str(tmp_path), nch, rows, False)
    b = Scan(ctx, str(tmp_path / "b"), nch, rows, False, extra=137, tables=a.tables)
    ssm = C.Ssm.generate(a.rp, ctx, C.SSM_BOTH)
    columns = [ssm.column(c) for c in (0, 4000, 4656)]
    for s in (a, b):
        s.rc.set_volume(ssm, None)
    last = [np.inf, np.inf]
    for turn in range(2):
        for i, s in enumerate((a, b)):
            for stage in (4, 6):
                s.rc.iterate(ssm, 1, _opts(stage))
                cost = s.check(ssm)
                assert cost < last[i]
                last[i] = cost
    for c, (idx, w) in zip((0, 4000, 4656), columns):
        i, v = ssm.column(c)
        assert np.array_equal(i, idx) and np.array_equal(v, w)


@pytest.mark.parametrize("nch,rows", [(48, 4), (47, 5)])
def test_changes_between_kernels(ctx, tmp_path, nch, rows):
    s = Scan(ctx, str(tmp_path), nch, rows, False)
    ssm = C.Ssm.generate(s.rp, ctx, C.SSM_BOTH)
    s.rc.set_volume(ssm, None)
    batch = C.Batch([s.rc], [ssm], ctx)
    last = np.inf
    for step in (4, 0, 6, 1, 4, "batch", 4, 3, 5, 4, "fp32", 6, "cta", 4, "sequential", 4):
        if step == "batch":
            batch.iterate(1, C.icd_opts(weights=C.SSM_FP16, warps_in_flight=256))
        elif step == "sequential":
            s.rc.iterate(ssm, 1, C.icd_opts(mode=C.ICD_SEQUENTIAL))
        elif step == "fp32":
            s.rc.iterate(ssm, 1, C.icd_opts(weights=C.SSM_FP32, warps_in_flight=256, lattice=16))
        elif step == "cta":
            s.rc.iterate(ssm, 1, C.icd_opts(weights=C.SSM_FP16, warps_per_voxel=8, warps_in_flight=2368, lattice=16))
        else:
            s.rc.iterate(ssm, 1, _opts(step, warps=4736 if step >= 4 else 256))
        cost = s.check(ssm)
        assert cost < last, step
        last = cost
