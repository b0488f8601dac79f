"""The work a user has this library do, as timed cases.

Each case is one call (or the few calls that belong together) through the
package's public entry points, on inputs made on the GPU from a seed.  The
kinds, and what each stands for:

* ``viewer``   an interactive viewer through the barney C API: the camera
               moved, so the accumulation is reset, one pass is rendered and
               the frame is read into host memory;
* ``frame``    a frame of several passes of a resident volume (offline or
               settled view), from any voxel store, with or without an
               iso-surface, or from a NanoVDB grid;
* ``batch``    many independent scenes of uneven sizes in one launch;
* ``ea_train`` one step of fitting a volume and a transfer function to
               images: the emission-absorption march, a loss, the adjoint;
* ``ea_view``  emission-absorption images without gradients;
* ``timestep`` a time-varying volume through the barney C API: texels come
               from host memory, the scene is rebuilt, rendered, read and
               released;
* ``ingest``   a new volume made ready to render on the device: voxel store,
               macrocells, majorants and the env light's tables, or a NanoVDB
               grid parsed, uploaded and its macrocells built.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from barney_gb300 import _native as N
from barney_gb300 import bn, scenes
from barney_gb300.batch import GpuBatch
from barney_gb300.device import GpuScene
from barney_gb300.ea import EAProblem, ea_render_autograd
from barney_gb300.nanovdb import GpuNanoVDBScene

_FMT = {"f32": N.GBV_VOXEL_F32, "f16": N.GBV_VOXEL_F16, "bf16": N.GBV_VOXEL_BF16, "u8": N.GBV_VOXEL_U8_SCALED}
_TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "u8": torch.uint8}
_READ = {"float4": bn.BN_FLOAT4, "rgba8": bn.BN_UFIXED8_RGBA, "srgb8": bn.BN_UFIXED8_RGBA_SRGB}
_MOST_PASSES = 1920 * 1080 * 12  # pixels x passes of a drawn frame


def listed():
    return [
        # the smallest call: a preview of a small volume, one pass of the default (single-scatter) build
        dict(name="viewer_64_preview", kind="viewer", nx=64, ny=64, nz=64, w=256, h=256, spp=1, multi=False,
             env=False, read="rgba8", fmt="f32"),
        # an ordinary interactive frame: multiple scattering under a sky, 720p
        dict(name="viewer_256_720p", kind="viewer", nx=256, ny=256, nz=256, w=1280, h=720, spp=1, multi=True,
             env=True, read="srgb8", fmt="f32"),
        # a thumbnail of the small scene: few pixels, more passes
        dict(name="frame_64_16spp", kind="frame", nx=64, ny=64, nz=64, w=256, h=256, spp=16, multi=False, env=False,
             fmt="f32", iso="none", grid="none"),
        # the benchmark's frame: 512^3, 1080p, 64 passes, up to 4 bounces, sky env map
        dict(name="frame_512_1080p_64spp", kind="frame", nx=512, ny=512, nz=512, w=1920, h=1080, spp=64, multi=True,
             env=True, fmt="f32", iso="none", grid="none"),
        # an odd-sized volume in the compact store, odd-sized window, default build
        dict(name="frame_u8_ragged", kind="frame", nx=301, ny=187, nz=233, w=853, h=479, spp=8, multi=False,
             env=False, fmt="u8", iso="none", grid="none"),
        # a quantized NanoVDB grid rendered as it is
        dict(name="frame_nanovdb_fp8", kind="frame", nx=160, ny=144, nz=128, w=960, h=540, spp=8, multi=True,
             env=True, fmt="f32", iso="none", grid="fp8"),
        # an iso-surface inside its volume
        dict(name="frame_iso_256", kind="frame", nx=256, ny=256, nz=256, w=960, h=540, spp=8, multi=True, env=True,
             fmt="f32", iso="first", grid="none"),
        # the batched workload: 64 volumes with sides in [32, 256], 8 passes each
        dict(name="batch_64_8spp", kind="batch", count=64, lo=32, hi=256, spp=8, fmt="f32"),
        # one step of volume reconstruction: 128^3, 32 views of 256x256, half-voxel steps
        dict(name="ea_train_128_32views", kind="ea_train", nx=128, ny=128, nz=128, views=32, w=256, h=256,
             voxels_per_step=0.5),
        # one large emission-absorption image from a half-precision store
        dict(name="ea_view_384_1080p", kind="ea_view", nx=384, ny=384, nz=384, views=1, w=1920, h=1080, fmt="f16",
             voxels_per_step=0.5),
        # the next time step of a simulation shown: 8-bit texels from host memory, a few passes, read back
        dict(name="timestep_256_u8texels", kind="timestep", nx=256, ny=256, nz=256, w=1280, h=720, spp=4, multi=True,
             env=True, read="float4", texels="u8", fmt="f32"),
        # a NanoVDB grid received and made ready to render
        dict(name="ingest_nanovdb_192", kind="ingest", nx=192, ny=192, nz=192, mc=16, fmt="f32", grid="float",
             env=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    side = _log_int(rng, lo, hi)
    if rng.random() < 0.4:
        return side, side, side
    return tuple(min(hi, max(lo, int(side * rng.uniform(0.6, 1.0)))) for _ in range(3))


def _window(rng, w_lo, w_hi):
    w = _log_int(rng, w_lo, w_hi)
    return w, max(8, int(w * rng.choice([1.0, 0.75, 0.5625])))


def draw(rng):
    kind = rng.choice(["viewer", "frame", "frame", "frame", "batch", "ea_train", "ea_view", "timestep", "ingest"])
    multi = rng.random() < 0.6
    if kind == "viewer":
        nx, ny, nz = _dims(rng, 32, 320)
        w, h = _window(rng, 128, 1920)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, w=w, h=h, spp=1, multi=multi, env=multi and rng.random() < 0.8,
                    read=rng.choice(["rgba8", "srgb8", "float4"]), fmt=rng.choice(["f32", "f32", "f16", "u8"]))
    if kind == "frame":
        w, h = _window(rng, 96, 1920)
        spp = max(1, min(_log_int(rng, 1, 64), _MOST_PASSES // (w * h)))
        grid = rng.choice(["none", "none", "none", "float", "fp4", "fp8", "fp16", "fpn"])
        iso = "none" if grid != "none" else rng.choice(["none", "none", "first", "after", "alone"])
        if iso != "none":
            spp = max(1, min(spp, _MOST_PASSES // (3 * w * h)))
        nx, ny, nz = _dims(rng, 32, 176 if grid != "none" else 448)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, w=w, h=h, spp=spp, multi=multi, env=multi and rng.random() < 0.8,
                    fmt="f32" if grid != "none" else rng.choice(["f32", "f16", "bf16", "u8", "linear"]), iso=iso,
                    grid=grid)
    if kind == "batch":
        lo = _log_int(rng, 24, 64)
        return dict(kind=kind, count=_log_int(rng, 4, 64), lo=lo, hi=rng.randint(2 * lo, 256), spp=_log_int(rng, 1, 16),
                    fmt=rng.choice(["f32", "f16", "u8"]))
    if kind == "ea_train":
        nx, ny, nz = _dims(rng, 24, 160)
        w, h = _window(rng, 48, 320)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, views=_log_int(rng, 1, 40), w=w, h=h,
                    voxels_per_step=round(rng.uniform(0.4, 1.0), 3))
    if kind == "ea_view":
        nx, ny, nz = _dims(rng, 48, 384)
        w, h = _window(rng, 96, 1920)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, views=1 if w > 640 else _log_int(rng, 1, 16), w=w, h=h,
                    fmt=rng.choice(["f32", "f16", "bf16", "u8", "linear"]),
                    voxels_per_step=round(rng.uniform(0.4, 1.0), 3))
    if kind == "timestep":
        nx, ny, nz = _dims(rng, 32, 256)
        w, h = _window(rng, 128, 1280)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, w=w, h=h, spp=_log_int(rng, 1, 8), multi=multi,
                    env=multi and rng.random() < 0.8, read=rng.choice(["rgba8", "srgb8", "float4"]),
                    texels=rng.choice(["f32", "u8", "u16"]), fmt=rng.choice(["f32", "f16", "u8"]))
    grid = rng.choice(["none", "none", "float", "fp8", "fp16"])
    nx, ny, nz = _dims(rng, 32, 192 if grid != "none" else 256)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, mc=16 if grid != "none" else rng.choice([8, 16]), grid=grid,
                fmt="f32" if grid != "none" else rng.choice(["f32", "f16", "bf16", "u8"]), env=rng.random() < 0.6)


# ------------------------------------------------------------------ inputs --

def _volume(dims, seed, blobs, noise, octaves, amplitude):
    """A (nz, ny, nx) float32 CUDA volume in [0, 1]: Gaussian blobs, white
    noise and value-noise octaves, as the package's host generator makes them."""
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    ax = [torch.linspace(0.0, 1.0, n, device="cuda") for n in (nz, ny, nx)]
    v = torch.zeros((nz, ny, nx), device="cuda")
    for _ in range(blobs):
        c, sig, amp = rng.uniform(0.0, 1.0, 3), rng.uniform(0.05, 0.2), rng.uniform(0.2, 1.0)
        gz, gy, gx = (torch.exp(-(x - float(k)) ** 2 / (2.0 * sig * sig)) for x, k in zip(ax, c))
        v += (float(amp) * gz)[:, None, None] * (gy[:, None] * gx[None, :])[None]
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 77)
    if noise:
        v += noise * torch.rand(v.shape, generator=g, device="cuda")
    for k in range(octaves):
        cells = 8 << k
        lattice = 2.0 * torch.rand((1, 1, cells + 1, cells + 1, cells + 1), generator=g, device="cuda") - 1.0
        v += amplitude * 2.0 ** -k * torch.nn.functional.interpolate(lattice, size=(nz, ny, nx), mode="trilinear",
                                                                     align_corners=True)[0, 0]
    return v.clamp_(0.0, 1.0)


def _field(case, seed):
    """The case's volume on the GPU: the fine-structured one of the frame
    workload from 96 voxels on, the plain one below."""
    dims = (case["nx"], case["ny"], case["nz"])
    if max(dims) >= 96:
        return _volume(dims, seed, 64, 0.05, 4, 0.1)
    return _volume(dims, seed, 8, 0.05, 0, 0.0)


def _spec(case, seed, shape, host=None):
    """The Scene record of a rendering case (its scalars: `host`, or a stand-in
    of the right shape when the voxels are already on the device)."""
    nz, ny, nx = shape
    rng = np.random.default_rng(seed + 5)
    scalars = host if host is not None else np.broadcast_to(np.float32(0), (nz, ny, nx))
    h = 1.0 / (max(nx, ny, nz) - 1)
    eye = np.array([0.3, 0.4, 1.0]) + rng.uniform(-0.15, 0.15, 3)
    eye *= 2.5 / np.linalg.norm(eye)
    big = max(nx, ny, nz) >= 96
    multi = bool(case.get("multi", False))
    sun = -1.0 / math.sqrt(3.0)
    s = scenes.Scene(scalars=scalars, tf=scenes.tf_two_peaks(256) if big else scenes.tf_ramp(128),
                     base_density=50.0 if big else 20.0, cells_per_mc=int(case.get("mc", 16 if big else 8)),
                     cam_pos=tuple(float(x) for x in eye), cam_dir=tuple(float(-x) for x in eye),
                     dir_lights=[((sun, sun, sun), (1.0, 1.0, 1.0), 2.0)],
                     env=scenes.env_sky(512, 256) if case.get("env") else None, ambient=0.3,
                     multi_scatter=int(multi), volume_multi_scatter=int(multi), max_volume_bounces=4 if multi else 0,
                     width=int(case.get("w", 64)), height=int(case.get("h", 64)), spp=int(case.get("spp", 1)),
                     origin=tuple(-0.5 * h * (n - 1) for n in (nx, ny, nz)), spacing=(h, h, h))
    iso = case.get("iso", "none")
    if iso != "none":
        s.iso = scenes.IsoSurface(value=0.5, color=(0.8, 0.7, 0.5, 1.0), instance=1 if iso == "after" else 0)
        s.volume_instance = 0 if iso in ("after", "alone") else 1
        s.no_volume = iso == "alone"
    return s


class _Session:
    """A barney context that gives its memory back when the state is dropped."""

    def __init__(self):
        self.s = bn.BarneySession(0)

    def __del__(self):
        try:
            self.s.close()
        except Exception:
            pass


def _read_buffer(case):
    shape = (case["h"], case["w"], 4) if case["read"] == "float4" else (case["h"], case["w"])
    return torch.empty(shape, dtype=torch.float32 if case["read"] == "float4" else torch.int32).pin_memory()


def _ea_setup(case, seed):
    dims = (case["nx"], case["ny"], case["nz"])
    vol = _volume(dims, seed, 16, 0.0, 0, 0.0)
    h = 1.0 / (max(dims) - 1)
    s = scenes.Scene(scalars=np.broadcast_to(np.float32(0), vol.shape), tf=scenes.tf_two_peaks(256),
                     base_density=20.0, cells_per_mc=8, origin=tuple(-0.5 * h * (n - 1) for n in dims),
                     spacing=(h, h, h))
    views = scenes.fibonacci_views(case["views"], 2.5, 8)
    for v in views:
        v["width"], v["height"] = case["w"], case["h"]
    return vol, s, views, float(case["voxels_per_step"]) * h


def _train_inputs(case, seed):
    vol, s, views, step = _ea_setup(case, seed)
    tf = torch.from_numpy(s.tf).cuda()
    with torch.no_grad():
        target = EAProblem(s, views, step, scalars=vol.reshape(-1), tf=tf).render()
    return s, views, step, (0.3 + 0.2 * vol).reshape(-1), tf, target


def _batch_scenes(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["count"] * 1000 + case["lo"])  # the items' sizes are the case's, not the seed's
    out = []
    for k in range(case["count"]):
        dims = [int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(3)]
        vol = _volume(dims, seed * 1000 + k, 8, 0.05, 0, 0.0)
        eye = rng.normal(size=3)
        eye *= 2.5 / np.linalg.norm(eye)
        size = int(sizes.choice([128, 256, 512]))
        sun = -1.0 / math.sqrt(3.0)
        out.append(scenes.Scene(scalars=vol.cpu().numpy(), tf=scenes.tf_two_ramps(128, rng), base_density=20.0,
                                cells_per_mc=8, cam_pos=tuple(float(x) for x in eye),
                                cam_dir=tuple(float(-x) for x in eye),
                                cam_up=(0.0, 1.0, 0.0) if abs(eye[1]) < 2.4 else (1.0, 0.0, 0.0),
                                dir_lights=[((sun, sun, sun), (1.0, 1.0, 1.0), 2.0)], ambient=0.3, width=size,
                                height=size, spp=case["spp"]))
    return out


def _gpu_scene(case, scene, vol):
    if case["fmt"] == "linear":
        return GpuScene(scene, layout=N.GBV_LAYOUT_LINEAR, scalars_device=vol.reshape(-1))
    return GpuScene(scene, fmt=_FMT[case["fmt"]], scalars_device=vol.reshape(-1))


def _grid_background(case, vol):
    """A copy of the volume with its faint part set to the grid's background,
    as sparse grids hold it."""
    return torch.where(vol < 0.05, torch.zeros_like(vol), vol).cpu().numpy()


def _grid_bytes(case, scene, host):
    h = scene.spacing[0]
    return scenes.nanovdb_grid(host, (0, 0, 0), h, tuple(float(o) - 0.5 * h for o in scene.origin), background=0.0,
                               grid_type=case["grid"], tolerance=0.01 if case["grid"] == "fpn" else -1.0)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind)
    if kind == "viewer":
        vol = _field(case, seed)
        host = vol.cpu().numpy()
        st["session"] = _Session()
        st["scene"] = _spec(case, seed, vol.shape, host)
        st["session"].s.build_scene(st["scene"], host.ctypes.data, voxel_format=_FMT[case["fmt"]],
                                    color_format=_READ[case["read"]])
        st["frame"] = _read_buffer(case)
    elif kind == "frame":
        vol = _field(case, seed)
        if case["grid"] != "none":
            host = _grid_background(case, vol)
            scene = _spec(case, seed, vol.shape, host)
            st["gpu"] = GpuNanoVDBScene(scene, _grid_bytes(case, scene, host))
        else:
            st["gpu"] = _gpu_scene(case, _spec(case, seed, vol.shape), vol)
        st["accum"] = st["gpu"].new_accum()
    elif kind == "batch":
        st["batch"] = GpuBatch(_batch_scenes(case, seed), fmt=_FMT[case["fmt"]])
    elif kind == "ea_train":
        s, views, step, scalars, tf, target = _train_inputs(case, seed)
        st["problem"] = EAProblem(s, views, step, scalars=scalars, tf=tf)
        st["scalars"], st["tf"] = scalars.clone().requires_grad_(True), tf.clone().requires_grad_(True)
        st["target"] = target
    elif kind == "ea_view":
        vol, s, views, step = _ea_setup(case, seed)
        if case["fmt"] == "linear":
            st["problem"] = EAProblem(s, views, step, scalars=vol.reshape(-1))
        else:
            store = _gpu_scene(case, s, vol)
            st["problem"] = EAProblem(s, views, step, scalars=store.scalars, store=store)
    elif kind == "timestep":
        vol = _field(case, seed)
        if case["texels"] == "f32":
            host = vol.cpu()
        else:
            top = 255 if case["texels"] == "u8" else 65535
            host = (vol * top).round().to(torch.int32).cpu().to(torch.uint8 if top == 255 else torch.uint16)
        st["texels"] = host.pin_memory()
        st["texel_format"] = {"f32": bn.BN_FLOAT32, "u8": bn.BN_UFIXED8, "u16": bn.BN_UFIXED16}[case["texels"]]
        st["scene"] = _spec(case, seed, vol.shape)
        st["session"] = _Session()
        st["frame"] = _read_buffer(case)
    elif kind == "ingest":
        vol = _field(case, seed)
        if case["grid"] != "none":
            host = _grid_background(case, vol)
            st["scene"] = _spec(case, seed, vol.shape, host)
            st["grid"] = _grid_bytes(case, st["scene"], host)
        else:
            st["scene"] = _spec(case, seed, vol.shape)
            st["scalars"] = vol.reshape(-1)
    else:
        raise ValueError(kind)
    return st


# --------------------------------------------------------------- the calls --

def run(st):
    case, kind = st["case"], st["kind"]
    if kind == "viewer":
        b = st["session"].s
        b.L.bnAccumReset(b.handles["fb"])
        b.render()
        return b.read(st["frame"])
    if kind == "frame":
        return st["gpu"].render(accum=st["accum"])
    if kind == "batch":
        st["batch"].render(case["spp"])
        return st["batch"].accums
    if kind == "ea_train":
        img = ea_render_autograd(st["scalars"], st["tf"], st["problem"])
        loss = ((img - st["target"]) ** 2).sum()
        gv, gt = torch.autograd.grad(loss, (st["scalars"], st["tf"]))
        return {"image": img.detach(), "grad_voxels": gv, "grad_tf": gt}
    if kind == "ea_view":
        return {"image": st["problem"].render()}
    if kind == "timestep":
        b = st["session"].s
        b.build_scene(st["scene"], st["texels"].data_ptr(), voxel_format=_FMT[case["fmt"]],
                      color_format=_READ[case["read"]], texel_format=st["texel_format"])
        b.render()
        out = b.read(st["frame"])
        b.release_scene()
        return out
    if case["grid"] != "none":
        g = GpuNanoVDBScene(st["scene"], st["grid"])
        return {"grid": g.grid, "ranges": g.ranges, "majorants": g.majorants, **_env_out(g)}
    g = GpuScene(st["scene"], fmt=_FMT[case["fmt"]], scalars_device=st["scalars"])
    out = {"store": g.voxels.view(_TORCH[case["fmt"]]), "ranges": g.ranges, "majorants": g.majorants, **_env_out(g)}
    if g.scale_offset is not None:
        out["scale_offset"] = g.scale_offset.view(torch.float32)
    return out


def _env_out(g):
    return {"cdf_y": g.cdf_y, "cdf_x": g.cdf_x} if g.cdf_y is not None else {}


# ---------------------------------------------------------- required work ---

def work(case):
    """Bytes: the voxels once in the form the case holds them, the outputs
    once.  Operations: per path, box test, a few cell steps, a sample and a
    shading; per march step, a trilinear sample, a transfer-function read and
    the compositing (twice as much again for its adjoint)."""
    kind = case["kind"]
    if kind == "batch":
        side = math.sqrt(case["lo"] * case["hi"])
        pixels = case["count"] * 256 * 256
        return {"bytes": case["count"] * side ** 3 * 4 + 16 * pixels, "flops": 300 * pixels * case["spp"]}
    voxels = case["nx"] * case["ny"] * case["nz"]
    size = {"f16": 2, "bf16": 2, "u8": 1}.get(case.get("fmt", "f32"), 4)
    size = {"fp4": 0.5, "fp8": 1, "fp16": 2, "fpn": 1}.get(case.get("grid", "none"), size)
    env = 512 * 256 * 16 if case.get("env") else 0
    if kind in ("ea_train", "ea_view"):
        pixels = case["views"] * case["w"] * case["h"]
        # a view of the unit cube from 2.5 away at 60 degrees: its box covers
        # about a fifth of the image's square, crossed over about 0.85 sides
        steps = case["views"] * 0.2 * case["h"] ** 2 * 0.85 * max(case["nx"], case["ny"], case["nz"]) / case[
            "voxels_per_step"]
        if kind == "ea_view":
            return {"bytes": size * voxels + 16 * pixels, "flops": 80 * steps}
        return {"bytes": 3 * 4 * voxels + 4 * 16 * pixels, "flops": 240 * steps}
    if kind == "ingest":
        mc = -(-case["nx"] // case["mc"]) * -(-case["ny"] // case["mc"]) * -(-case["nz"] // case["mc"])
        store = 8 * size * voxels if case["grid"] == "none" else size * voxels
        return {"bytes": 4 * voxels + store + 12 * mc + env, "flops": 4 * voxels}
    pixels = case["w"] * case["h"]
    out = 4 if case.get("read") in ("rgba8", "srgb8") else 16
    if kind == "timestep":
        size = 8 * size + {"f32": 4, "u8": 1, "u16": 2}[case["texels"]]
    return {"bytes": size * voxels + out * pixels + env, "flops": 300 * pixels * case["spp"]}


# --------------------------------------------- the same in 64-bit arithmetic --

def exact(case, seed):
    """The march and its gradients, and the tables of an ingest, in float64.
    Delta-tracked frames have no such value: they are sums over random paths."""
    if case["kind"] in ("ea_train", "ea_view"):
        return _exact_ea(case, seed)
    if case["kind"] == "ingest" and case["grid"] in ("none", "float"):
        return _exact_ingest(case, seed)
    return None


def _rays(view):
    """Pixel-centre rays of a perspective view: (eye, directions (h*w, 3))."""
    def unit(v):
        return v / np.linalg.norm(v)
    d = unit(np.asarray(view["dir"], np.float64))
    du = unit(np.cross(d, np.asarray(view["up"], np.float64)))
    dv = unit(np.cross(du, d))
    d = d / (2.0 * math.tan(0.5 * view["fovy"] * math.pi / 180.0))
    w, h = view["width"], view["height"]
    u = torch.tensor((np.arange(w) + 0.5) / w - 0.5, device="cuda") * (w / h)
    v = torch.tensor((np.arange(h) + 0.5) / h - 0.5, device="cuda")
    t = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    r = t(d) + u[None, :, None] * t(du) + v[:, None, None] * t(dv)
    return t(np.asarray(view["pos"], np.float64)), (r / r.norm(dim=-1, keepdim=True)).reshape(-1, 3)


def _march(vol, tf, scene, view, step, each):
    """Runs `each` for every march step of a view with (ray indices, corner
    indices (8, k), corner weights (8, k), tf index, tf fraction, clamped)."""
    nz, ny, nx = vol.shape
    eye, dirs = _rays(view)
    lo = torch.tensor(np.float32(scene.origin).astype(np.float64), device="cuda")
    h = torch.tensor(np.float32(scene.spacing).astype(np.float64), device="cuda")
    cells = torch.tensor([nx - 1, ny - 1, nz - 1], device="cuda", dtype=torch.float64)
    a, b = (lo - eye) / dirs, (lo + h * cells - eye) / dirs
    t0 = torch.minimum(a, b).amax(-1).clamp_min(0.0)
    t1 = torch.maximum(a, b).amin(-1)
    hit = torch.nonzero(t0 < t1)[:, 0]
    t0, t1, dirs = t0[hit], t1[hit], dirs[hit]
    order = torch.argsort(t1 - t0, descending=True)
    hit, t0, t1, dirs = hit[order], t0[order], t1[order], dirs[order]
    if hit.numel() == 0:
        return
    length = ((t1 - t0) / step).cpu().numpy()
    flat, n = vol.reshape(-1), tf.shape[0]
    for i in range(int(math.ceil(length[0] - 0.5))):
        k = int(np.searchsorted(-length, -(i + 0.5), side="left"))  # rays with t0 + (i + 1/2) step < t1
        if k == 0:
            break
        rel = (eye + (t0[:k] + (i + 0.5) * step)[:, None] * dirs[:k] - lo) / h
        inside = ((rel >= 0) & (rel < cells)).all(-1)
        rel = torch.minimum(rel.clamp_min(0.0), cells)
        c = torch.minimum(rel.floor(), cells - 1.0)
        f = rel - c
        c = c.long()
        base = c[:, 0] + nx * (c[:, 1] + ny * c[:, 2])
        at = torch.stack([base + (q & 1) + nx * ((q >> 1) & 1) + nx * ny * (q >> 2) for q in range(8)])
        wt = torch.stack([(f[:, 0] if q & 1 else 1 - f[:, 0]) * (f[:, 1] if q & 2 else 1 - f[:, 1]) *
                          (f[:, 2] if q & 4 else 1 - f[:, 2]) for q in range(8)])
        s = (flat[at] * wt).sum(0)  # domain (0, 1)
        clamped = ~((s > 0) & (s < 1))
        g = s.clamp(0.0, 1.0) * (n - 1)
        idx = g.long().clamp_max(n - 2)
        each(hit[:k], at, wt, idx, g - idx, clamped, inside)


def _exact_ea(case, seed):
    if case["kind"] == "ea_train":
        scene, views, step, scalars, tf, target = _train_inputs(case, seed)
        vol = scalars.reshape(case["nz"], case["ny"], case["nx"]).double()
    else:
        vol, scene, views, step = _ea_setup(case, seed)
        if case["fmt"] == "u8":
            return None  # the store's own 8-bit codes
        vol = vol.to(_TORCH.get(case["fmt"], torch.float32)).double()
        tf = torch.from_numpy(scene.tf).cuda()
    step = float(np.float32(step))
    tf = tf.double()
    rho, n = float(np.float32(scene.base_density)), tf.shape[0]
    images, gvol, gtf = [], torch.zeros(vol.numel(), dtype=torch.float64, device="cuda"), torch.zeros_like(tf)
    for at_view, view in enumerate(views):
        px = view["width"] * view["height"]
        color = torch.zeros((px, 3), dtype=torch.float64, device="cuda")
        tau = torch.zeros(px, dtype=torch.float64, device="cuda")

        def forward(ray, at, wt, idx, f, clamped, inside):
            m = (1 - f)[:, None] * tf[idx] + f[:, None] * tf[idx + 1]
            x = torch.where(inside, m[:, 3] * rho * step, torch.zeros_like(f))
            color[ray] += (torch.exp(-tau[ray]) * -torch.expm1(-x))[:, None] * m[:, :3]
            tau[ray] += x

        _march(vol, tf, scene, view, step, forward)
        img = torch.cat([color, -torch.expm1(-tau)[:, None]], dim=1)
        images.append(img)
        if case["kind"] == "ea_view":
            continue
        g = 2.0 * (img - target[at_view * px:(at_view + 1) * px].double())
        done, depth, end = torch.zeros_like(color), torch.zeros_like(tau), torch.exp(-tau)

        def backward(ray, at, wt, idx, f, clamped, inside):
            e0, e1 = tf[idx], tf[idx + 1]
            m = (1 - f)[:, None] * e0 + f[:, None] * e1
            x = torch.where(inside, m[:, 3] * rho * step, torch.zeros_like(f))
            w = torch.exp(-depth[ray]) * -torch.expm1(-x)
            done[ray] += w[:, None] * m[:, :3]
            depth[ray] += x
            after = torch.exp(-depth[ray])
            q = g[ray]
            dx = q[:, 3] * end[ray] + (q[:, :3] * (m[:, :3] * after[:, None] - (color[ray] - done[ray]))).sum(-1)
            dm = torch.cat([q[:, :3] * w[:, None], (dx * step * rho)[:, None]], dim=1)
            dm = torch.where(inside[:, None], dm, torch.zeros_like(dm))
            gtf.index_add_(0, idx, dm * (1 - f)[:, None])
            gtf.index_add_(0, idx + 1, dm * f[:, None])
            ds = (dm * (e1 - e0)).sum(-1) * (n - 1)
            k = torch.nonzero((ds != 0) & ~clamped)[:, 0]
            gvol.index_add_(0, at[:, k].reshape(-1), (wt[:, k] * ds[k]).reshape(-1))

        _march(vol, tf, scene, view, step, backward)
    image = torch.cat(images)
    if case["kind"] == "ea_view":
        return {"image": image}
    return {"image": image, "grad_voxels": gvol, "grad_tf": gtf}


def _windows(v, first, last, dim, reduce):
    return torch.stack([reduce(v.narrow(dim, a, b - a + 1), dim) for a, b in zip(first, last)], dim=dim)


def _exact_ingest(case, seed):
    vol = _field(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["grid"] == "float":  # macrocell m covers [m size / mc, (m + 1) size / mc + 1], background around the voxels
        values = torch.nn.functional.pad(torch.where(vol < 0.05, torch.zeros_like(vol), vol).double(), (0, 2) * 3)
        first = [[m * n // -(-n // 16) for m in range(-(-n // 16))] for n in (nx, ny, nz)]
        last = [[(m + 1) * n // -(-n // 16) + 1 for m in range(-(-n // 16))] for n in (nx, ny, nz)]
    else:
        if case["fmt"] == "u8":
            return None  # the store's own 8-bit codes
        values = vol.to(_TORCH[case["fmt"]]).double()
        mcs = [-(-(n - 1) // case["mc"]) for n in (nx, ny, nz)]
        first = [[m * case["mc"] for m in range(k)] for k in mcs]
        last = [[min(n - 1, (m + 1) * case["mc"]) for m in range(k)] for n, k in zip((nx, ny, nz), mcs)]
    lo = hi = values
    for axis, dim in ((0, 2), (1, 1), (2, 0)):
        lo = _windows(lo, first[axis], last[axis], dim, lambda t, d: t.amin(d))
        hi = _windows(hi, first[axis], last[axis], dim, lambda t, d: t.amax(d))
    scene = _spec(case, seed, vol.shape)
    alpha = torch.from_numpy(scene.tf[:, 3]).cuda().double()
    n = alpha.numel()
    g = [x.reshape(-1).clamp(0.0, 1.0) * (n - 1) for x in (lo, hi)]
    idx = [x.long().clamp_max(n - 2) for x in g]
    ends = [(1 - (x - i)) * alpha[i] + (x - i) * alpha[i + 1] for x, i in zip(g, idx)]
    top = torch.maximum(*ends)
    for i in range(n):
        top = torch.where((idx[0] < i) & (i <= idx[1]), top.clamp_min(float(alpha[i])), top)
    out = {"ranges": torch.stack([lo.reshape(-1), hi.reshape(-1)], dim=1).reshape(-1),
           "majorants": top * scene.base_density}
    if case["grid"] == "none":
        out["store"] = _exact_store(values, vol.shape)
    else:
        out["grid"] = None  # bytes
    if scene.env is not None:
        out.update(_exact_env(scene.env))
    return out


def _exact_store(values, shape):
    """8^3-cell bricks, x fastest; each cell its 8 corners; zeros past the last cell."""
    nz, ny, nx = shape
    nb = [-(-(k - 1) // 8) for k in (nz, ny, nx)]
    cells = torch.stack([values[dz:nz - 1 + dz, dy:ny - 1 + dy, dx:nx - 1 + dx]
                         for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)], dim=-1)
    pad = torch.zeros((nb[0] * 8, nb[1] * 8, nb[2] * 8, 8), dtype=torch.float64, device="cuda")
    pad[:nz - 1, :ny - 1, :nx - 1] = cells
    return pad.reshape(nb[0], 8, nb[1], 8, nb[2], 8, 8).permute(0, 2, 4, 1, 3, 5, 6).reshape(-1)


def _exact_env(env):
    """A texel's weight: the largest channel over the 3 x 3 bilinear reads at
    its corners, edge midpoints and centre (x wraps, y clamps)."""
    t = torch.from_numpy(env.texels[..., :3]).cuda().double()
    rows = [0.5 * (torch.cat([t[:1], t[:-1]]) + t), t, 0.5 * (t + torch.cat([t[1:], t[-1:]]))]
    weight = torch.zeros(t.shape[:2], dtype=torch.float64, device="cuda")
    for r in rows:
        for c in (0.5 * (r.roll(1, 1) + r), r, 0.5 * (r + r.roll(-1, 1))):
            weight = torch.maximum(weight, c.amax(-1))
    line = weight.cumsum(1)
    theta = math.pi * (torch.arange(t.shape[0], device="cuda", dtype=torch.float64) + 0.5) / t.shape[0]
    col = (line[:, -1] * torch.sin(theta)).cumsum(0)
    return {"cdf_y": col / col[-1], "cdf_x": (line / line[:, -1:]).reshape(-1)}
