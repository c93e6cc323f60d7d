"""Measured cases: the work a user of this framework has it do, each through a
public entry point (the Python stage functions and objects, and the C ABI's
device-to-device rotation), over the sizes its workloads, tests and benchmark
run.

Kinds of a case:
  icd         grouped ICD iterations, image copied back: either a scan's raw
              data (on the device) from a zero image, or the next iterations
              of a reconstruction under way (start="image")
  resume      the same from an initial image (FP64 forward projection), with
              the exact FP64 cost after every iteration (the stopping rule)
  sequential  the icd_iteration stage with host buffers in the reference's
              visiting order (the stage function's default)
  batch       several uneven scans advanced together
  matrix      a new geometry: stored system matrix and reconstruction state,
              then one iteration from an initial image
  rotate      rotating-to-fixed slice rotation, device to device
  predict     forward pass of the warm-start network
  train       one training step of it: gradients of a few crops, Adam
"""
from __future__ import annotations

import atexit
import ctypes as C
import math
import os
import random
import shutil
import tempfile

import numpy as np
import torch

import ctbb_icd_b200 as CB
from ctbb_icd_b200 import learned as L
from ctbb_icd_b200 import replicas as R
from ctbb_icd_b200 import workloads as W
from ctbb_icd_b200._lib import check, lib, ptr

MU = W.MU_WATER
_DIR = None


def listed():
    return [
        # Smallest call: the test suite's 32 x 32 x 6 scan, where launches and
        # latency count; default options, edge-preserving, flying focal spot.
        dict(name="icd small", kind="icd", workload="small_ffs", iters=3, weights="fp32"),
        # An ordinary reduced scan with default options: 128 x 128 x 16, quadratic.
        dict(name="icd ordinary", kind="icd", workload="cfg1", iters=2, weights="fp32"),
        # The warm start's early iterations: half-size grid of the benchmark
        # scan, FP16 matrix, one warp per update, its fixed visiting order.
        dict(name="icd early", kind="icd", workload="cfg2_train", iters=1, weights="fp16", lattice=32, warps=4096,
             start="image"),
        # Odd and ragged: 201 x 201 x 37, 40 rows, no flying focal spot,
        # quadratic, settings as the autotuner picks them for FP16.
        dict(name="icd ragged", kind="icd", nx=201, nz=37, rows=40, row_iso=0.06, ffs=False, pitch=0.9, fov=21.3,
             penalty="quadratic", iters=1, weights="fp16", stage=4, wpv=8, warps=4736, lattice=32,
             start="image"),
        # The benchmark: 512 x 512 x 64, FP16 matrix, the autotuned settings.
        dict(name="icd full", kind="icd", workload="cfg2", iters=1, weights="fp16", stage=4, wpv=8, warps=4736,
             lattice=128, start="image"),
        # Continuing from an image with the exact-cost stopping rule.
        dict(name="resume", kind="resume", workload="cfg2_lite", iters=2, weights="fp16", stage=4, wpv=8, warps=0,
             lattice=0),
        # The drop-in stage with its defaults: reference order, host buffers.
        dict(name="sequential", kind="sequential", workload="cfg1_small", iters=1),
        # Uneven independent scans in one launch per iteration.
        dict(name="batch", kind="batch", scans=4, spec_seed=3, max_nx=256, max_nz=24, iters=1),
        # A new protocol: matrix build and first iteration of a scan on the
        # benchmark's scanner, voxels near the training grid's.
        dict(name="matrix", kind="matrix", nx=160, nz=8, rows=64, row_iso=0.06, ffs=True, pitch=1.0, fov=24.0,
             penalty="edge-preserving", iters=1, weights="fp16"),
        # End of every reconstruction: the full volume to the fixed frame.
        dict(name="rotate", kind="rotate", nx=512, nz=64, direction=-1),
        # The learned start on its training grid.
        dict(name="predict", kind="predict", nx=256, ny=256, nz=32),
        # One step of its training: crops of 8 x 128 x 128.
        dict(name="train", kind="train", nx=128, ny=128, nz=8, crops=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["icd", "icd", "icd", "icd", "resume", "sequential", "batch", "matrix", "rotate", "predict",
                       "train"])
    if kind == "rotate":
        return dict(kind=kind, nx=_log_int(rng, 32, 512), nz=rng.randint(1, 64), direction=rng.choice([-1, 1]))
    if kind == "predict":
        return dict(kind=kind, nx=_log_int(rng, 24, 256), ny=_log_int(rng, 24, 256), nz=rng.randint(4, 32))
    if kind == "train":
        return dict(kind=kind, nx=_log_int(rng, 40, 144), ny=_log_int(rng, 40, 144), nz=rng.randint(4, 12),
                    crops=rng.randint(1, 3))
    if kind == "batch":
        return dict(kind=kind, scans=rng.randint(2, 5), spec_seed=rng.randint(0, 10000), max_nx=256,
                    max_nz=rng.randint(10, 24), iters=1)
    rows = rng.choice([8, 16, 32, 40, 64])
    g = dict(kind=kind, rows=rows, row_iso=0.06 if rows >= 32 else 0.12, ffs=rng.random() < 0.5,
             pitch=round(rng.uniform(0.6, 1.4), 3), penalty=rng.choice(["quadratic", "edge-preserving"]))
    if kind == "sequential":
        return dict(g, nx=_log_int(rng, 16, 44), nz=rng.randint(2, 6), fov=round(rng.uniform(21.5, 30.0), 2), iters=1)
    g.update(nx=_log_int(rng, 48, 224 if kind == "icd" else 112), nz=rng.randint(3, 40 if kind == "icd" else 16),
             fov=round(rng.uniform(21.5, 30.0), 2), iters=rng.randint(1, 2))
    if kind == "icd":
        g["start"] = rng.choice(["zero", "image"]) if g["penalty"] == "quadratic" else "image"
        if rng.random() < 0.5:
            return dict(g, weights=rng.choice(["fp32", "fp16"]))
    if rng.random() < 0.4:
        return dict(g, weights="fp32")
    return dict(g, weights="fp16", stage=4, wpv=8, warps=0, lattice=0)


# ---------------------------------------------------------------------------
# Geometry, phantom images, options
# ---------------------------------------------------------------------------
def _prm(case):
    if "workload" in case:
        return W.workload(case["workload"])["prm"]
    rows, row_iso, pitch, nx, nz, ffs = (case[k] for k in ("rows", "row_iso", "pitch", "nx", "nz", "ffs"))
    feed, vz = pitch * rows * row_iso, row_iso
    turns = int(math.ceil((nz * vz + 2.6 * rows * row_iso) / feed)) + 2
    quad = case["penalty"] == "quadratic"
    z_start = 0.1 * feed * 10.0 - 0.5 * turns * feed + 0.5 * nz * vz
    prm = {**W._BASE, **W._scanner(736, 366.25, W.FAN_INC, rows, row_iso, 1152, ffs, pitch, turns),
           **W._recon(nx, case["fov"], vz, nz, z_start, case["penalty"], 1e3 if quad else 0.1,
                      0.005 if quad else 9.6e-4, 10)}
    return prm


def _configure(prm):
    global _DIR
    if _DIR is None:
        _DIR = tempfile.mkdtemp(prefix="ctbb_cases_")
        atexit.register(shutil.rmtree, _DIR, ignore_errors=True)
        open(os.path.join(_DIR, "raw.bin"), "wb").close()
    prm = dict(prm, sinogram_path=os.path.join(_DIR, "raw.bin"), output_dir=_DIR, output_file="out.img")
    return CB.configure_recon_params(W.write_prm(os.path.join(_DIR, "case.prm"), prm))


def _scan(case_prm, seed):
    """Parameters, slice tables and the raw frames of the water phantom with
    its six inserts, Poisson noise, from the device projector."""
    ctx = CB.default_context()
    rp = _configure(case_prm)
    tables = CB.slice_tables(rp)
    spec = W.phantom_spec(dict(n_ellipsoids=0, seed=seed, i0_lo=5e4, i0_hi=2e5))
    spec.clip_z_lo, spec.clip_z_hi = W.slab_clip(rp, tables.slice_locations)
    raw = torch.empty(rp.raw_shape, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    check(lib().ctbb_gpu_synth_raw(ctx.handle, C.byref(rp.geom), C.byref(spec), C.c_void_p(raw.data_ptr())))
    return ctx, rp, tables, raw


def _iterate(rp, tables, seed):
    """The image of a reconstruction of that scan under way: the phantom in
    each slice's rotating frame with 1 % noise, float32 [nz][ny][nx]."""
    g = rp.geom
    nz, ny, nx = rp.shape
    gen = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31))
    x = ((torch.arange(nx, device="cuda") - g.center_voxel_x) * g.voxel_size_x)[None, None, :]
    y = ((torch.arange(ny, device="cuda") - g.center_voxel_y) * g.voxel_size_y)[None, :, None]
    a = torch.tensor([2.0 * math.pi / g.num_views_per_turn * float(i) for i in tables.slice_indices], device="cuda")
    c, s = a.cos()[:, None, None], a.sin()[:, None, None]
    px, py = c * x - s * y, s * x + c * y
    vol = MU * (px * px + py * py < 100.0).float()
    for i, hu in enumerate((-200.0, -100.0, -50.0, 50.0, 100.0, 1000.0)):
        b = i * math.pi / 3.0
        vol += MU * hu / 1000.0 * ((px - 6.0 * math.cos(b)) ** 2 + (py - 6.0 * math.sin(b)) ** 2 < 2.25)
    vol *= 1 + 0.01 * torch.randn(vol.shape, generator=gen, device="cuda")
    return vol.clamp_min(0).cpu().numpy()


def _image(nx, ny, nz, seed):
    """An attenuation image [nz][ny][nx] (cm^-1): a water disc with random
    discs in it, 1 % noise, air outside."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31))
    y = torch.linspace(-1, 1, ny, device="cuda")[:, None]
    x = torch.linspace(-1, 1, nx, device="cuda")[None, :]
    body = (x * x + y * y < 0.45).float()
    par = torch.rand(12, 4, generator=g, device="cuda")
    img = MU * body
    for cx, cy, r, v in par.tolist():
        d = (x - cx + 0.5) ** 2 + (y - cy + 0.5) ** 2 < (0.03 + 0.15 * r) ** 2
        img = img + MU * (1.2 * v - 0.3) * d * body
    vol = img[None] * (1 + 0.01 * torch.randn(nz, ny, nx, generator=g, device="cuda"))
    return vol.clamp_min(0).contiguous()


def _opts(case, **more):
    w = CB.SSM_FP16 if case["weights"] == "fp16" else CB.SSM_FP32
    return CB.icd_opts(weights=w, lattice=case.get("lattice", 0), warps_in_flight=case.get("warps", 0),
                       stage_column=case.get("stage", 0), warps_per_voxel=case.get("wpv", 1), **more)


def _batch_specs(case):
    specs = [s for s in R.batch_specs(64, case["spec_seed"])]
    out = []
    for s in specs:
        p = s["prm"]
        nz = int(round(abs(p["z_end"] - p["z_start"]) / p["slice_thickness"] - 0.5))
        if p["nx"] <= case["max_nx"] and nz <= case["max_nz"] and len(out) < case["scans"]:
            out.append(p)
    return out


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    ctx = CB.default_context()
    if kind == "rotate":
        n, nz = case["nx"], case["nz"]
        rp = _configure(dict(W.workload("cfg2")["prm"], nx=n, ny=n, z_end=-3.0 - (nz + 0.5) * 0.06))
        s = dict(kind=kind, ctx=ctx, rp=rp, tables=CB.slice_tables(rp), vol=_image(n, n, rp.shape[0], seed),
                 direction=case["direction"])
        return dict(s, out=torch.empty_like(s["vol"]))
    if kind == "predict":
        return dict(kind=kind, net=CB.WarmStartNet.load(ctx), x=_image(case["nx"], case["ny"], case["nz"], seed))
    if kind == "train":
        crops = []
        for i in range(case["crops"]):
            xc = _image(case["nx"], case["ny"], case["nz"], 100 * seed + i)
            g = torch.Generator(device="cuda").manual_seed((100 * seed + i) % (1 << 31))
            x = (xc + 0.02 * torch.randn(xc.shape, generator=g, device="cuda")).clamp_min(0)
            crops.append((x, xc, (xc > 0).float()))
        return dict(kind=kind, net=CB.WarmStartNet(ctx, L.DEFAULT_BLOCKS, seed=seed % 1000), crops=crops)
    if kind == "batch":
        scans = []
        for i, prm in enumerate(_batch_specs(case)):
            _, rp, tables, raw = _scan(prm, 100 * seed + i)
            scans.append((CB.Recon(rp, tables.slice_indices, ctx), CB.Ssm.generate(rp, ctx, CB.SSM_FP32), raw))
        return dict(kind=kind, scans=scans, iters=case["iters"], opts=CB.icd_opts(),
                    batch=CB.Batch([s[0] for s in scans], [s[1] for s in scans], ctx))
    _, rp, tables, raw = _scan(_prm(case), seed)
    s = dict(kind=kind, ctx=ctx, rp=rp, tables=tables, iters=case["iters"])
    if kind == "sequential":
        data = CB.CtData(raw=raw.cpu().numpy(), tube_angles=tables.tube_angles, slice_indices=tables.slice_indices)
        CB.generate_system_matrix(rp, data, ctx, CB.SSM_FP32)
        return dict(s, data=data)
    s.update(raw=raw, opts=_opts(case))
    if kind in ("resume", "matrix") or case.get("start") == "image":
        s["x0"] = _iterate(rp, tables, seed)
    if kind == "resume":
        s["opts"] = _opts(case, stop_rel_change=1e-12)
    if kind != "matrix":
        s["rc"] = CB.Recon(rp, tables.slice_indices, ctx)
        s["ssm"] = CB.Ssm.generate(rp, ctx, CB.SSM_FP16 if case["weights"] == "fp16" else CB.SSM_FP32)
    if kind == "icd" and "x0" in s:
        s["rc"].set_raw_device(raw.data_ptr())
        s["rc"].set_volume(s["ssm"], s["x0"])
        s["under_way"] = True
    return s


def run(s):
    kind = s["kind"]
    if kind == "rotate":
        t = s["tables"]
        check(lib().ctbb_gpu_rotate_device(s["ctx"].handle, C.byref(s["rp"].geom), ptr(t.tube_angles, C.c_double),
                                           ptr(t.slice_indices, C.c_uint64), C.c_void_p(s["vol"].data_ptr()),
                                           C.c_void_p(s["out"].data_ptr()), s["direction"]))
        return s["out"]
    if kind == "predict":
        return s["net"].forward(s["x"])
    if kind == "train":
        net = s["net"]
        loss = [net.accumulate_gradient(*c) for c in s["crops"]]
        grad = net.gradient()
        net.adam_step(1e-4, grad_scale=1.0 / len(loss))
        return dict(loss=loss, gradient=grad, params=net.params())
    if kind == "batch":
        for rc, ssm, raw in s["scans"]:
            rc.set_raw_device(raw.data_ptr())
            rc.set_volume(ssm, None)
        st = s["batch"].iterate(s["iters"], s["opts"])
        return dict(volumes=[rc.volume() for rc, _, _ in s["scans"]], updates=int(st.voxel_updates))
    if kind == "sequential":
        d = s["data"]
        d.recon_volume = np.zeros(s["rp"].shape, np.float32)
        CB.icd_iteration(s["rp"], d, s["ctx"], n_iter=s["iters"])
        return dict(volume=d.recon_volume, volume_f64=d.extra["volume_f64"])
    if kind == "matrix":
        ssm = CB.Ssm.generate(s["rp"], s["ctx"], CB.SSM_BOTH)
        rc = CB.Recon(s["rp"], s["tables"].slice_indices, s["ctx"])
        rc.set_raw_device(s["raw"].data_ptr())
        rc.set_volume(ssm, s["x0"])
        rc.iterate(ssm, s["iters"], s["opts"])
        info = ssm.info()
        out = dict(volume=rc.volume(), nnz=int(info.nnz), longest=int(info.max_col_nnz))
        rc.free()
        ssm.free()
        return out
    rc = s["rc"]
    if not s.get("under_way"):
        rc.set_raw_device(s["raw"].data_ptr())
        rc.set_volume(s["ssm"], s.get("x0"))
    st = rc.iterate(s["ssm"], s["iters"], s["opts"])
    out = dict(volume=rc.volume(), updates=int(st.voxel_updates))
    if kind == "resume":
        out["cost"] = st.cost
    return out


# ---------------------------------------------------------------------------
# work / exact
# ---------------------------------------------------------------------------
def _sizes(prm):
    """(matrix entries, voxels, sinogram samples, updates' entries) of a scan.
    A voxel column meets about 2 v / (channel pitch at its distance) channels
    and 2 vz / (row pitch) rows per view, 0.9 for the mean obliquity and 0.8
    for the views whose rows leave the detector."""
    rp = _configure(prm)
    CB.slice_tables(rp)
    g = rp.geom
    nz, ny, nx = rp.shape
    ch = max(1.0, 2 * 0.9 * g.voxel_size_x / (g.focal_spot_radius * W.FAN_INC))
    rows = max(1.0, 2 * g.voxel_size_z / prm["CollSlicewidth"])
    per_col = g.num_views_for_system_matrix * ch * rows * 0.8
    return per_col * nx * ny, nx * ny * nz, float(np.prod(rp.raw_shape)), per_col * nx * ny * nz


def work(case):
    kind = case["kind"]
    if kind == "rotate":
        n = case["nx"] ** 2 * case["nz"]
        return dict(bytes=8 * n, flops=20 * n)
    if kind in ("predict", "train"):
        n = case["nx"] * case["ny"] * case["nz"]
        blocks = L.DEFAULT_BLOCKS
        fwd = 2 * 27 * n * (2 * 32 + 2 * blocks * 32 * 32)
        params = 4 * (27 * 32 + 32 + 2 * blocks * (27 * 1024 + 32) + 27 * 32 + 1)
        if kind == "predict":
            return dict(bytes=8 * n + params, flops=fwd)
        return dict(bytes=case["crops"] * 12 * n + 8 * params, flops=case["crops"] * 3 * fwd)
    if kind == "batch":
        b = f = 0.0
        for prm in _batch_specs(case):
            nnz, nvox, nsino, ent = _sizes(prm)
            b += case["iters"] * (8 * nnz + 8 * nsino + 8 * nvox) + 4 * nsino
            f += case["iters"] * 6 * ent
        return dict(bytes=b, flops=f)
    nnz, nvox, nsino, ent = _sizes(_prm(case))
    per_entry = 6 if case.get("weights") == "fp16" else 8
    wide = 2 if kind == "sequential" else 1  # FP64 image and estimate
    b = case["iters"] * (per_entry * nnz + 8 * wide * nsino + 8 * wide * nvox) + 4 * nsino
    f = case["iters"] * 6 * ent
    if kind == "resume":  # A x for the start and after each iteration
        b += (case["iters"] + 1) * (per_entry * nnz + 8 * nsino + 4 * nvox)
        f += (case["iters"] + 1) * 2 * ent
    if kind == "matrix":  # both weight formats written, then A x
        b += 10 * nnz + per_entry * nnz + 8 * nsino + 4 * nvox
        f += 40 * nnz + 2 * ent
    return dict(bytes=b, flops=f)


def _net64(p, blocks, x, s_in):
    """The network in 64 bits: x [nz][ny][nx] -> prediction of that shape."""
    conv = torch.nn.functional.conv3d
    at = [0]

    def take(*shape):
        n = math.prod(shape)
        t = p[at[0]:at[0] + n].reshape(shape)
        at[0] += n
        return t

    def layer(a, ci, co):
        w = take(27, ci, co).permute(2, 1, 0).reshape(co, ci, 3, 3, 3)
        return conv(a, w, take(co), padding=1)

    a = torch.relu(layer((s_in * x)[None, None], 1, 32))
    for _ in range(blocks):
        h = torch.relu(layer(a, 32, 32))
        a = a + layer(h, 32, 32)
    return layer(a, 32, 1)[0, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "rotate":
        s = prepare(case, seed)
        g, t, vol = s["rp"].geom, s["tables"], s["vol"].double()
        nz, n, _ = vol.shape
        idx = torch.arange(n, dtype=torch.float64, device="cuda")
        x, y = (idx - g.center_voxel_x)[None, :], (idx - g.center_voxel_y)[:, None]
        out = torch.zeros_like(vol)
        for k in range(nz):
            a = s["direction"] * math.radians(float(t.tube_angles[int(t.slice_indices[k])]))
            u = math.cos(a) * x - math.sin(a) * y + g.center_voxel_x
            v = math.sin(a) * x + math.cos(a) * y + g.center_voxel_y
            ok = (u >= 0) & (u <= n - 2) & (v >= 0) & (v <= n - 2)
            i, j = u.clamp(0, n - 2).floor().long(), v.clamp(0, n - 2).floor().long()
            fu, fv = u - i, v - j
            p = vol[k]
            val = (p[j, i] * (1 - fu) * (1 - fv) + p[j, i + 1] * fu * (1 - fv) + p[j + 1, i] * (1 - fu) * fv
                   + p[j + 1, i + 1] * fu * fv)
            out[k] = torch.where(ok, val, torch.zeros_like(val))
        return out
    if kind == "predict":
        s = prepare(case, seed)
        p = torch.from_numpy(s["net"].params()).cuda().double()
        with torch.no_grad():
            return _net64(p, s["net"].blocks, s["x"].double(), s["net"].scaling()[0])
    if kind == "train":
        s = prepare(case, seed)
        s_in, s_out = s["net"].scaling()
        p = torch.from_numpy(s["net"].params()).cuda().double().requires_grad_(True)
        loss = []
        for x, xc, m in s["crops"]:
            r = _net64(p, s["net"].blocks, x.double(), s_in) - (xc.double() - x.double()) * s_out
            loss.append((m.double() * r * r).sum() / m.double().sum())
            loss[-1].backward()
        return dict(loss=[float(v) for v in loss], gradient=p.grad.cpu().numpy(), params=None)
    return None  # iterates of a concurrent (or sequential) descent have no closed form
