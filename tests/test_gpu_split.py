"""Frames whose tiles are handed out pass by pass (their fragments logged and
added up by a second kernel) equal frames rendered whole, bit for bit.

gbv_render splits every tile that may see the field while the log has room;
gbv_render_noalloc has no log and splits none.  The sizes are the edges: one
pixel, part of a warp tile, one tile, one tile and a column and a row, and
frames whose log has room for part of the tiles or for none."""
import ctypes as C
import subprocess
import threading
from pathlib import Path

import numpy as np
import pytest

from barney_gb300 import _native as N
from barney_gb300 import scenes
from barney_gb300.batch import GpuBatch
from barney_gb300.device import GpuScene, _ptr, _stream
import oracle

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def whole(g, spp, start=0, accum=None):
    acc = g.new_accum() if accum is None else accum
    N.check(N.lib().gbv_render_noalloc(C.byref(g.record()), _ptr(acc), g.s.width, g.s.height, start, spp, None,
                                       _stream()), "gbv_render_noalloc")
    return acc


def world(kind, w, h):
    """single / multi (isotropic) / forward (strong forward scattering, hits
    bounded by the path depth only) / dark (negative background alpha: the
    gradient) / iso / inside (camera in the volume: no tile is outside) /
    away (the frame sees nothing of it) / tele (a pixel spans less than the
    rectangle's margin allows)."""
    s = scenes.small_scene(dims=40, spp=1, width=w, height=h)
    if kind in ("multi", "forward", "inside_forward", "iso"):
        s.multi_scatter = s.volume_multi_scatter = 1
        s.max_volume_bounces = 4
        s.env = scenes.env_sky(64, 32)
    if kind.endswith("forward"):
        s.anisotropy, s.max_volume_bounces = 0.8, 20
    if kind == "dark":
        s.bg_color = (0.5, 0.25, 0.125, -1.0)
    if kind == "iso":
        s.iso, s.volume_instance = scenes.IsoSurface(value=0.5), 1
    if kind.startswith("inside"):
        s.cam_pos = (0.05, 0.02, 0.03)
    if kind == "away":
        s.cam_dir = tuple(-x for x in s.cam_dir)
    if kind == "tele":
        s.fovy = 0.05
    return s


KINDS = ["single", "multi", "forward", "dark", "iso", "inside", "away", "tele"]


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (8, 4), (9, 5), (57, 33)])
@pytest.mark.parametrize("kind", KINDS)
def test_split_equals_whole(cuda, kind, size):
    """Fresh frames (the first pass overwrites) and continued ones, 1 pass and
    several."""
    import torch
    g = GpuScene(world(kind, *size))
    for spp, start in ((1, 0), (5, 0), (3, 2)):
        base = torch.rand(size[1], size[0], 4, device="cuda")
        a = g.render(spp=spp, accum=base.clone(), accum_id_start=start)
        b = whole(g, spp, start, base.clone())
        torch.cuda.synchronize()
        np.testing.assert_array_equal(bits(a.cpu().numpy()), bits(b.cpu().numpy()))


@pytest.mark.parametrize("kind", ["single", "dark", "inside", "away"])
def test_split_frames_are_the_oracles(cuda, kind):
    import torch
    s = world(kind, 41, 23)
    a = GpuScene(s).render(spp=4)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(bits(a.cpu().numpy()), bits(oracle.Oracle(s).render(spp=4)))


@pytest.mark.parametrize("kind,w,h,spp,start", [("inside", 640, 400, 220, 0), ("forward", 320, 200, 130, 3),
                                                ("inside_forward", 1280, 800, 5, 0), ("inside", 200, 120, 2000, 0)])
def test_frames_larger_than_the_log_equal_whole(cuda, kind, w, h, spp, start):
    """Frames rendered in parts of as many passes as the log holds (the first
    two, whose last parts are shorter), and one whose log does not hold enough
    passes of all tiles, which splits part of them."""
    import torch
    g = GpuScene(world(kind, w, h))
    base = torch.rand(h, w, 4, device="cuda")
    a, b = g.render(spp=spp, accum=base.clone(), accum_id_start=start), whole(g, spp, start, base.clone())
    torch.cuda.synchronize()
    np.testing.assert_array_equal(bits(a.cpu().numpy()), bits(b.cpu().numpy()))


def test_split_batch_equals_whole(cuda):
    """Items with and without outer tiles, with other bounds on their hits."""
    import torch
    sizes = [(1, 1), (9, 5), (57, 33), (64, 40), (16, 8)]
    items = [world(k, *sizes[i % 5]) for i, k in enumerate(["single", "multi", "forward", "inside", "away", "dark"])]
    b = GpuBatch(items)
    for spp, start in ((1, 0), (5, 1)):
        b.render(spp, accum_id_start=start)
    for s, acc in zip(items, b.accums):
        g = GpuScene(s)
        ref = whole(g, 5, 1, whole(g, 1))
        torch.cuda.synchronize()
        np.testing.assert_array_equal(bits(acc.cpu().numpy()), bits(ref.cpu().numpy()))


def test_scratch_is_safe_across_threads_and_streams(cuda):
    """Launches on several threads and streams share the scratch pool: every
    frame is the one a lone launch renders."""
    import torch
    gs = [GpuScene(world("single", 40 + 8 * i, 30)) for i in range(4)]
    refs = [whole(g, 6).cpu().numpy() for g in gs]
    out = [None] * 4
    torch.cuda.synchronize()

    def work(i):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            frames = [gs[i].render(spp=6) for _ in range(8)]
        st.synchronize()
        out[i] = [f.cpu().numpy() for f in frames]

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for ref, frames in zip(refs, out):
        for f in frames:
            np.testing.assert_array_equal(bits(f), bits(ref))


def test_threads_render_scenes_of_other_tables(cuda, tmp_path):
    """Threads render scenes whose shared-memory tables differ in size (few
    and many macrocells, without an env map and with low and high ones,
    without tables at all): no call fails, and every frame is the one a lone
    launch renders."""
    import torch
    root = Path(__file__).resolve().parent.parent
    lib = tmp_path / "librender_threads.so"
    r = subprocess.run(["gcc", "-std=c99", "-O2", "-fPIC", "-shared", "-I", str(root / "include"),
                        str(root / "tests" / "c" / "render_threads.c"), "-L", str(root / "barney_gb300" / "_lib"),
                        "-lbarney_gb300", f"-Wl,-rpath,{root / 'barney_gb300' / '_lib'}", "-lpthread", "-o", str(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    gs = []
    for dims, cells, env in ((16, 8, 0), (64, 2, 0), (16, 8, 1000), (64, 2, 32), (48, 4, 300), (64, 2, 0)):
        s = scenes.small_scene(dims=dims, spp=1, width=16, height=8)
        s.cells_per_mc = cells
        if env:
            s.env = scenes.env_sky(64, env)
        gs.append(GpuScene(s))
    n = len(gs)
    refs = [whole(g, 1).cpu().numpy() for g in gs]
    accums, streams = [g.new_accum() for g in gs], [torch.cuda.Stream() for _ in gs]
    torch.cuda.synchronize()
    records = [g.record() for g in gs]
    message = C.create_string_buffer(256)
    failed = C.CDLL(str(lib)).render_threads(
        (N.GbvScene * n)(*records), (C.c_void_p * n)(*[a.data_ptr() for a in accums]),
        (C.c_void_p * n)(*[st.cuda_stream for st in streams]), N.ivec(*[0] * (n - 1), 1), n, 16, 8, 2000, message)
    torch.cuda.synchronize()
    assert failed == 0, (failed, message.value.decode())
    for a, ref in zip(accums, refs):
        np.testing.assert_array_equal(bits(a.cpu().numpy()), bits(ref))


def test_captured_render_replays(cuda):
    """A render captured in a CUDA graph (its scratch belongs to the graph)
    replays to the same frame."""
    import torch
    g = GpuScene(world("single", 57, 33))
    ref = whole(g, 3)
    acc = g.new_accum()
    g.render(spp=3, accum=acc)  # loads the kernels outside the capture
    acc.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        with torch.cuda.graph(graph, stream=st):
            g.render(spp=3, accum=acc)
    for _ in range(2):
        acc.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(bits(acc.cpu().numpy()), bits(ref.cpu().numpy()))


@pytest.mark.parametrize("kind", ["single", "dark", "multi"])
def test_background_taken_in_groups_equals_wavefront(cuda, kind):
    """A frame with more background tiles than the GPU has warps twice over
    (they are taken several at a time), ragged at its right and lower edge,
    alone and in a batch of two, against the wavefront mode."""
    import torch
    s = world(kind, 2043, 1301)
    s.fovy = 120.0
    g = GpuScene(s)
    ref = g.render(spp=3, config={"mode": N.GBV_RENDER_WAVEFRONT})
    acc = g.render(spp=3)
    batch = GpuBatch([s, s])
    batch.render(3)
    torch.cuda.synchronize()
    for a in [acc, whole(g, 3)] + list(batch.accums):
        np.testing.assert_array_equal(bits(a.cpu().numpy()), bits(ref.cpu().numpy()))


@pytest.mark.parametrize("kind", ["single", "multi", "iso"])
@pytest.mark.parametrize("counted", [True, False])
def test_warps_that_give_up_are_reported(cuda, kind, counted):
    """The frame kernel's limit on a warp's looks for work, set so low that
    warps reach it while other warps' paths are under way: the frame may lack
    pixels, and the launch says so; with the limit out of reach it does not."""
    import torch
    g = GpuScene(world(kind, 640, 360))
    ref = g.render(spp=4)
    for polls in (0, 1 << 20):
        acc = g.new_accum()
        counters = torch.zeros(N.GBV_NUM_COUNTERS, dtype=torch.int64, device="cuda") if counted else None
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        N.check(N.lib().gbv_selftest_idle_limit(C.byref(g.record()), _ptr(acc), 640, 360, 4, polls, _ptr(counters),
                                                _ptr(flag), _stream()), "gbv_selftest_idle_limit")
        torch.cuda.synchronize()
        assert flag.item() == (polls == 0)
        if counted:
            assert (counters[N.GBV_COUNTER_CAPS].item() > 0) == (polls == 0)
        if polls:
            np.testing.assert_array_equal(bits(acc.cpu().numpy()), bits(ref.cpu().numpy()))


@pytest.mark.parametrize("turn", [60.0, 89.0, 95.0, 135.0, 180.0])
@pytest.mark.parametrize("fovy", [60.0, 170.0])
def test_field_beside_and_behind_the_camera(cuda, turn, fovy):
    """The camera turned away from the field, which is then partly or wholly
    behind it: the frame is the oracle's."""
    import torch
    s = world("dark", 41, 23)
    s.fovy = fovy
    d, a = np.array(s.cam_dir, float), np.radians(turn)
    side = np.cross(d, s.cam_up)
    s.cam_dir = tuple(np.cos(a) * d + np.sin(a) * side * np.linalg.norm(d) / np.linalg.norm(side))
    acc = GpuScene(s).render(spp=3)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(bits(acc.cpu().numpy()), bits(oracle.Oracle(s).render(spp=3)))
