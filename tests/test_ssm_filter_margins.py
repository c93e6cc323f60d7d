"""The matrix builder's FP32 filter (ssm.cu chan_filter), restated in numpy float32 and
checked on the CPU at the benchmark's geometry and with each flying focal spot, against the
entries of the oracle's ray-driven builder for sampled columns over every view of the window:
every entry lies in the rows that the filter leaves open, and every row that it calls certain
is an entry, so that the builder's counting and filling passes agree. The margins are derived
(four roundings of the lengths involved, four times over); with a quarter of them it still
holds."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import ctbb_icd_b200 as C  # noqa: E402
from ctbb_icd_b200 import workloads as W  # noqa: E402
import oracle_util as O  # noqa: E402
from test_ssm_bounds import CASES, view_tables  # noqa: E402

F = np.float32


def _margins(g, tables):
    cx, cy = abs(g.center_voxel_x) + int(g.num_voxels_x), abs(g.center_voxel_y) + int(g.num_voxels_y)
    reach = 2.0 * (g.focal_spot_radius + g.voxel_size_x * cx + g.voxel_size_y * cy)
    rows = abs(g.center_row) + int(g.Nrows_projection)
    slope = 2.0 * (rows * abs(g.axial_detector_spacing) + np.abs(tables["off2"]).max()) / g.source_detector_distance
    ulp = 16.0 / 16777216.0
    tol = 1e-3 + ulp * (reach / min(g.voxel_size_x, g.voxel_size_y) + cx + cy)
    zmax = np.abs(tables["src2"]).max()
    return tol, 1e-3 + ulp * ((zmax + reach * slope) / g.voxel_size_z + abs(g.center_voxel_z))


def chan_filter(g, tables, col, ch, v, share):
    """Open rows [r_lo, r_hi] and certain rows [s_lo, s_hi] of channels `ch` and views `v`."""
    tol, tolz = (F(share * m) for m in _margins(g, tables))
    V = {k: a.astype(F)[v] for k, a in tables.items()}
    nx, ny, nr = int(g.num_voxels_x), int(g.num_voxels_y), int(g.Nrows_projection)
    ic, jc = col % nx, col // nx
    xc, yc = F((ic - g.center_voxel_x) * g.voxel_size_x), F((jc - g.center_voxel_y) * g.voxel_size_y)
    ffs, sdd = bool(g.Phiffs or g.Zffs), g.source_detector_distance
    tang = (ch - g.center_channel_non_ffs) * (g.fan_angle_increment if ffs else g.transaxial_detector_spacing / sdd)
    A, B = (-sdd * np.cos(tang)).astype(F), (sdd * np.sin(tang)).astype(F)
    D0 = (A * V["ew0"] - B * V["eu0"]) - V["off0"]
    D1 = (A * V["ew1"] - B * V["eu1"]) - V["off1"]
    a0, a1 = np.abs(D0), np.abs(D1)
    xm = a0 > a1
    t = np.where(xm, xc - V["src0"], yc - V["src1"]) / np.where(xm, D0, D1)
    open_all = (np.abs(a0 - a1) <= F(1e-4) * np.maximum(a0, a1)) | ~(np.abs(t) > F(1e-6))
    u = (np.where(xm, V["src1"], V["src0"]) + np.where(xm, D1, D0) * t) * np.where(
        xm, F(1.0 / g.voxel_size_y), F(1.0 / g.voxel_size_x)) + np.where(xm, F(g.center_voxel_y), F(g.center_voxel_x))
    own, n = np.where(xm, jc, ic), np.where(xm, ny, nx)
    lo, hi = np.maximum(own - 1, 0).astype(F), np.minimum(own + 1, n - 1).astype(F)
    ivz, sa = F(1.0 / g.voxel_size_z), F(g.axial_detector_spacing)
    sz = t * ivz
    z0 = (V["src2"] * ivz + F(g.center_voxel_z)) + (F(g.center_row) * sa - V["off2"]) * sz
    rdz = F(-1) / (sa * sz)
    k0, k1 = (F(-1) - z0) * rdz, (F(1) - z0) * rdz
    ka, kb, d = np.minimum(k0, k1), np.maximum(k0, k1), tolz * np.abs(rdz) + F(share * 1e-3)
    assert u.dtype == z0.dtype == d.dtype == F
    out = (u < lo - tol) | (u > hi + tol)
    r_lo = np.where(open_all, 0, np.maximum(np.ceil(ka - d), 0)).astype(int)
    r_hi = np.where(open_all, nr - 1, np.where(out, -1, np.minimum(np.floor(kb + d), nr - 1))).astype(int)
    sure = ~open_all & ~out & (u > lo + tol) & (u < hi - tol) & (d < nr - 1)
    s_lo = np.where(sure, np.clip(np.ceil(ka + d), 0, nr), 0).astype(int)
    s_hi = np.where(sure, np.clip(np.floor(kb - d), -1, nr - 1), -1).astype(int)
    return r_lo, r_hi, s_lo, s_hi


@pytest.mark.parametrize("share", [1.0, 0.25])
@pytest.mark.parametrize("case", list(CASES))
def test_filter_decides_as_the_reference(tmp_path, case, share):
    name, overrides = CASES[case]
    _, rp = W.materialise(name, str(tmp_path), raw=False, overrides=overrides)
    C.slice_tables(rp)
    g = rp.geom
    nx, ny, nch, nr = (int(x) for x in (g.num_voxels_x, g.num_voxels_y, g.n_channels, g.Nrows_projection))
    nvsm = int(g.num_views_for_system_matrix)
    tables = view_tables(g, bool(g.Phiffs or g.Zffs))
    rng = np.random.default_rng(77)
    cols = np.unique(np.concatenate([[nx // 2 + nx * (ny // 2), 3 + nx * (ny // 2), nx // 4 + nx * (ny // 4)],
                                     rng.integers(0, nx * ny, 9)])).astype(np.int64)
    ref = O.port_ssm_subset(rp, cols, np.arange(nvsm, dtype=np.int32))
    certain = entries = 0
    for c in cols:
        q = ref[int(c)][0].astype(np.int64)
        if q.size == 0:
            continue
        v, ch, row = q // (nch * nr), (q // nr) % nch, q % nr
        r_lo, r_hi, _, _ = chan_filter(g, tables, int(c), ch, v, share)
        assert ((row >= r_lo) & (row <= r_hi)).all(), (case, int(c))
        # certain rows of every channel near the entries' own, and the entries among them
        known = np.zeros((nvsm, nch, nr), bool)
        known[v, ch, row] = True
        near = np.unique(np.concatenate([v * nch + np.clip(ch + k, 0, nch - 1) for k in range(-4, 5)]))
        vs, cs = near // nch, near % nch
        _, _, s_lo, s_hi = chan_filter(g, tables, int(c), cs, vs, share)
        for i in np.flatnonzero(s_hi >= s_lo):
            assert known[vs[i], cs[i], s_lo[i]: s_hi[i] + 1].all(), (case, int(c), int(vs[i]), int(cs[i]))
            certain += int(s_hi[i] - s_lo[i] + 1)
        entries += q.size
    assert entries > 20000 and certain > 0.5 * entries
