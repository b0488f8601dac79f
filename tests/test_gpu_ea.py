"""Fixed-step emission-absorption march and its adjoint on the GPU.

Tolerances: forward images within 1e-5 relative (plus 1e-6 absolute for
near-zero channels) of the oracle; the FP32 adjoint within 1e-3 relative
(norm over the checked entries) of central finite differences of the FP64
GPU march (eps = 1e-3) and of the oracle's FP64 gradient.
"""
import numpy as np
import pytest

from barney_gb300 import _native as N
from barney_gb300 import scenes
from barney_gb300.ea import EAProblem
import oracle

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-5, 1e-6


def small_problem(dims=48, nviews=6, size=48):
    gt = scenes.ea_scene(dims)
    views = scenes.fibonacci_views(nviews, 2.5, size)
    step = 0.5 / (dims - 1)
    return gt, views, step


def test_forward_matches_oracle(cuda):
    gt, views, step = small_problem()
    p = EAProblem(gt, views, step)
    img = p.render().cpu().numpy().reshape(-1, 4)
    o = oracle.Oracle(gt)
    ref32 = o.ea_render(views, step)
    ref64 = o.ea_render(views, step, use_double=True)
    np.testing.assert_allclose(img, ref32, rtol=RTOL, atol=ATOL)
    # FP32 against FP64: rounding of sample positions, trilinear weights and
    # steep TF segments; measured max ~3e-4 relative on 0.2% of channels
    np.testing.assert_allclose(img, ref64, rtol=1e-3, atol=1e-5)
    assert img[:, 3].max() > 0.5


def test_forward_f64_matches_oracle(cuda):
    gt, views, step = small_problem(nviews=3)
    p = EAProblem(gt, views, step)
    img = p.render_f64().cpu().numpy().reshape(-1, 4)
    ref64 = oracle.Oracle(gt).ea_render(views, step, use_double=True)
    np.testing.assert_allclose(img, ref64, rtol=1e-6, atol=1e-7)


def test_constant_density_beer_lambert(cuda):
    """Known answer: a constant field maps to constant (rgb, sigma); a pixel
    whose march takes n steps gives A = 1-exp(-n sigma dt), C = rgb*A."""
    vol = np.full((16, 16, 16), 0.5, np.float32)
    tf = np.tile(np.array([[0.2, 0.6, 0.9, 0.4]], np.float32), (4, 1))
    s = scenes.Scene(scalars=vol, tf=tf, base_density=3.0)
    views = [dict(pos=(0.0, 0.0, 2.5), dir=(0.0, 0.0, -1.0), up=(0.0, 1.0, 0.0), fovy=20.0, width=8, height=8)]
    step = 0.01
    img = EAProblem(s, views, step).render().cpu().numpy().reshape(8, 8, 4)
    # central pixels: the ray runs along -z through the whole box (t0=2, t1=3)
    sigma = 0.4 * 3.0
    t0, t1 = 2.0, 3.0
    n = sum(1 for i in range(200) if t0 + (i + 0.5) * step < t1)
    a = 1 - np.exp(-n * sigma * step)
    c = img[3, 3]
    np.testing.assert_allclose(c[3], a, rtol=2e-5)
    np.testing.assert_allclose(c[:3], np.array([0.2, 0.6, 0.9]) * a, rtol=2e-5)


@pytest.mark.parametrize("tf_kind", ["ramp", "two_peaks"])
def test_adjoint_matches_oracle_and_finite_differences(cuda, tf_kind):
    """The two-peak TF has knots (slope changes) inside the data range, where a
    central difference averages two one-sided slopes; the finite-difference
    check therefore runs on the knot-free ramp TF, and both TFs are checked
    against the oracle's FP64 gradient."""
    import torch
    gt, views, step = small_problem(dims=40, nviews=4, size=40)
    if tf_kind == "ramp":
        gt.tf = scenes.tf_ramp(256, 0.9)
    p_gt = EAProblem(gt, views, step)
    target = p_gt.render()
    start = scenes.Scene(scalars=np.full_like(gt.scalars, 0.3) + 0.2 * gt.scalars, tf=gt.tf,
                         base_density=gt.base_density)
    p = EAProblem(start, views, step)
    img = p.render()
    gimg = 2.0 * (img - target)  # dL/dI of L = sum (I - target)^2
    gv, gt_tf = p.backward(img, gimg)
    gv, gt_tf = gv.cpu().numpy().astype(np.float64), gt_tf.cpu().numpy().astype(np.float64)
    # FP64 oracle gradient
    o = oracle.Oracle(start)
    ov, ot = o.ea_backward(views, step, gimg.cpu().numpy().reshape(-1, 4))
    ov = ov.reshape(-1)
    sel = np.flatnonzero(np.abs(ov) > 1e-3 * np.abs(ov).max())
    assert np.linalg.norm(gv.reshape(-1)[sel] - ov[sel]) <= 1e-3 * np.linalg.norm(ov[sel])
    assert np.linalg.norm(gt_tf - ot) <= 1e-3 * np.linalg.norm(ot)
    if tf_kind != "ramp":
        return
    # central finite differences of the FP64 march, eps = 1e-3
    rng = np.random.default_rng(44)
    tgt64 = target.double()

    def loss(pp):
        return float(((pp.render_f64() - tgt64) ** 2).sum().item())

    def fd_of(make, base, eps=1e-3):
        hi, lo = np.float32(base + eps), np.float32(base - eps)
        return (loss(make(float(hi))) - loss(make(float(lo)))) / (float(hi) - float(lo))

    vox = rng.choice(sel, size=16, replace=False)
    base = start.scalars.reshape(-1)
    fd = np.array([fd_of(lambda x, v=v: p.with_voxel(int(v), x), float(base[v])) for v in vox])
    an = gv.reshape(-1)[vox]
    assert np.linalg.norm(fd - an) <= 1e-3 * np.linalg.norm(fd) + 1e-6, (fd, an)
    tsel = np.flatnonzero(np.abs(ot.reshape(-1)) > 1e-3 * np.abs(ot).max())
    ent = rng.choice(tsel, size=min(16, tsel.size), replace=False)
    tfb = start.tf.reshape(-1)
    fd = np.array([fd_of(lambda x, e=e: p.with_tf_entry(int(e), x), float(tfb[e])) for e in ent])
    an = gt_tf.reshape(-1)[ent]
    assert np.linalg.norm(fd - an) <= 1e-3 * np.linalg.norm(fd) + 1e-6, (fd, an)


def test_autograd_function(cuda):
    import torch
    from barney_gb300.ea import ea_render_autograd
    gt, views, step = small_problem(dims=32, nviews=2, size=32)
    p = EAProblem(gt, views, step)
    vox = p.scalars.clone().requires_grad_(True)
    tf = p.tf.clone().requires_grad_(True)
    img = ea_render_autograd(vox, tf, p)
    w = torch.rand_like(img)
    (img * w).sum().backward()
    gv, gtf = p.backward(img.detach(), w)
    # the adjoint's atomics sum in no fixed order: equal up to FP32 reassociation
    torch.testing.assert_close(vox.grad.reshape(-1), gv.reshape(-1), rtol=1e-4, atol=1e-6)
    torch.testing.assert_close(tf.grad.reshape(-1), gtf.reshape(-1), rtol=1e-4, atol=1e-5)


def _rounded(v, fmt):
    if fmt == N.GBV_VOXEL_F16:
        return v.astype(np.float16).astype(np.float32)
    u = v.view(np.uint32).astype(np.uint64)
    u = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16
    return u.astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("fmt,brick", [(N.GBV_VOXEL_F32, (3, 3, 3)), (N.GBV_VOXEL_F32, (4, 2, 2)),
                                       (N.GBV_VOXEL_F16, (3, 3, 3)), (N.GBV_VOXEL_BF16, (2, 2, 2))])
def test_forward_on_brick_stores(cuda, fmt, brick):
    """The forward march over a brick-corner store equals the march over the
    linear FP32 field holding the same (rounded) voxel values, bit for bit."""
    from barney_gb300.device import GpuScene
    gt, views, step = small_problem(nviews=3)
    g = GpuScene(gt, fmt=fmt, brick=brick)
    got = EAProblem(gt, views, step, store=g).render().cpu().numpy()
    rounded = gt.scalars if fmt == N.GBV_VOXEL_F32 else _rounded(gt.scalars, fmt)
    import copy
    gr = copy.copy(gt)
    gr.scalars = np.ascontiguousarray(rounded)
    ref = EAProblem(gr, views, step).render().cpu().numpy()
    np.testing.assert_array_equal(got.view(np.uint32), ref.view(np.uint32))


def test_forward_on_u8_store_error_against_fp64(cuda):
    from barney_gb300.device import GpuScene
    gt, views, step = small_problem(nviews=3)
    g = GpuScene(gt, fmt=N.GBV_VOXEL_U8_SCALED)
    got = EAProblem(gt, views, step, store=g).render().cpu().numpy().reshape(-1, 4)
    ref64 = oracle.Oracle(gt).ea_render(views, step, use_double=True)
    err = np.abs(got - ref64)
    # 8-bit voxels per 8^3 cells: a few 1e-3 on the image
    assert float(np.sqrt(np.mean(err ** 2))) < 5e-3 and err.max() < 0.05, (np.sqrt(np.mean(err ** 2)), err.max())


def test_forward_on_u8_store_matches_oracle_u8_form(cuda):
    """Against the oracle's U8 storage form the U8 forward agrees as closely
    as the FP32 forward does with the FP32 oracle."""
    from barney_gb300.device import GpuScene
    gt, views, step = small_problem(nviews=3)
    g = GpuScene(gt, fmt=N.GBV_VOXEL_U8_SCALED)
    got = EAProblem(gt, views, step, store=g).render().cpu().numpy().reshape(-1, 4)
    ref = oracle.Oracle(gt, u8=True).ea_render(views, step)
    np.testing.assert_allclose(got, ref, rtol=RTOL, atol=ATOL)


def test_adjoint_rejects_brick_stores(cuda):
    import ctypes as C
    from barney_gb300.device import GpuScene, _ptr, _stream
    gt, views, step = small_problem(nviews=1)
    g = GpuScene(gt, fmt=N.GBV_VOXEL_F16)
    p = EAProblem(gt, views, step, store=g)
    rec = p.record()
    rec.d_voxels = g.voxels.data_ptr()
    rec.format, rec.layout = g.fmt, g.layout
    import torch
    img = p.render()
    gv = torch.zeros(p.scalars.numel(), device="cuda")
    gtf = torch.zeros(p.tf.numel(), device="cuda")
    st = N.lib().gbv_ea_backward(C.byref(rec), p._views_c, 1, step, _ptr(img), _ptr(img), _ptr(gv), _ptr(gtf),
                                 _stream())
    assert st == N.GBV_ERROR_UNSUPPORTED


def test_reconstruction_loop_reduces_the_loss(cuda):
    """The differentiable workload in miniature: a density grid that starts
    at a constant 0.1 and the transfer function are fitted to target views
    of a blob volume by Adam steps through the autograd wrapper (at 0.1 the
    two-peak TF is flat zero, so the first gradients reach the TF entries);
    the L2 loss falls well below its start."""
    import torch
    from barney_gb300.ea import ea_render_autograd
    gt = scenes.ea_scene(24)
    views = scenes.fibonacci_views(8, 2.5, 24)
    step = 0.5 / 23
    target = EAProblem(gt, views, step).render()
    start = scenes.Scene(scalars=np.full_like(gt.scalars, 0.1), tf=gt.tf, base_density=gt.base_density)
    p = EAProblem(start, views, step)
    vox = p.scalars.clone().requires_grad_(True)
    tf = p.tf.clone().requires_grad_(True)
    opt = torch.optim.Adam([vox, tf], lr=0.02)
    losses = []
    for _ in range(40):
        opt.zero_grad()
        img = ea_render_autograd(vox, tf, p)
        loss = ((img - target) ** 2).mean()
        loss.backward()
        opt.step()
        with torch.no_grad():
            vox.clamp_(0.0, 1.0)
            tf.clamp_(0.0, 1.0)
        losses.append(float(loss.item()))
    assert losses[-1] < 0.3 * losses[0], losses[::8]


def test_differentiable_workload_at_its_named_size(cuda):
    """The differentiable emission-absorption workload at its own size: a
    128^3 FP32 density grid, the 256-entry two-peak TF, 32 views of 256^2 on
    a Fibonacci sphere of radius 2.5, step 0.5 voxel, L2 loss against target
    views of the seeded ground-truth blob volume.
    - forward: within 1e-5 relative (+1e-6 absolute) of the FP32 oracle;
    - adjoint: within 1e-3 relative (norm over entries above 1e-3 of the
      largest) of the oracle's FP64 gradient, voxels and TF entries;
    - central finite differences (eps = 1e-3) of the FP64 GPU march at 64
      random voxels and 64 random TF entries (seed 44): within 1e-3
      relative.  The FD check runs on the knot-free ramp TF (a central
      difference across a TF knot averages two one-sided slopes; see
      test_adjoint_matches_oracle_and_finite_differences), with the same
      grid, views, step and loss."""
    import torch
    dims = 128
    gt = scenes.ea_scene(dims)
    views = scenes.fibonacci_views(32, 2.5, 256)
    assert len(views) == 32 and all(v["width"] == v["height"] == 256 for v in views)
    step = 0.5 / (dims - 1)
    for tf_kind in ("two_peaks", "ramp"):
        truth = gt if tf_kind == "two_peaks" else scenes.Scene(scalars=gt.scalars, tf=scenes.tf_ramp(256, 0.9),
                                                                base_density=gt.base_density,
                                                                cells_per_mc=gt.cells_per_mc)
        target = EAProblem(truth, views, step).render()
        # parameters away from the truth, where every gradient term is live
        start = scenes.Scene(scalars=np.full_like(truth.scalars, 0.3) + 0.2 * truth.scalars, tf=truth.tf,
                             base_density=truth.base_density, cells_per_mc=truth.cells_per_mc)
        p = EAProblem(start, views, step)
        img = p.render()
        o = oracle.Oracle(start)
        if tf_kind == "two_peaks":
            np.testing.assert_allclose(img.cpu().numpy(), o.ea_render(views, step), rtol=RTOL, atol=ATOL)
        gimg = 2.0 * (img - target)
        gv, gtf = p.backward(img, gimg)
        torch.cuda.synchronize()
        gv = gv.cpu().numpy().astype(np.float64)
        gtf = gtf.cpu().numpy().astype(np.float64).reshape(-1)
        ov, ot = o.ea_backward(views, step, gimg.cpu().numpy().reshape(-1, 4))
        ov, ot = ov.reshape(-1), ot.reshape(-1)
        sel = np.flatnonzero(np.abs(ov) > 1e-3 * np.abs(ov).max())
        tsel = np.flatnonzero(np.abs(ot) > 1e-3 * np.abs(ot).max())
        assert sel.size > 10000 and tsel.size >= 64, (sel.size, tsel.size)
        assert np.linalg.norm(gv[sel] - ov[sel]) <= 1e-3 * np.linalg.norm(ov[sel])
        assert np.linalg.norm(gtf[tsel] - ot[tsel]) <= 1e-3 * np.linalg.norm(ot[tsel])
        if tf_kind != "ramp":
            continue
        rng = np.random.default_rng(44)
        tgt64 = target.double()

        def loss(pp):
            return float(((pp.render_f64() - tgt64) ** 2).sum().item())

        def fd_of(make, base, eps=1e-3):
            hi, lo = np.float32(base + eps), np.float32(base - eps)
            return (loss(make(float(hi))) - loss(make(float(lo)))) / (float(hi) - float(lo))

        vox = rng.choice(sel, size=64, replace=False)
        base = start.scalars.reshape(-1)
        fd = np.array([fd_of(lambda x, v=v: p.with_voxel(int(v), x), float(base[v])) for v in vox])
        an = gv[vox]
        assert np.linalg.norm(fd - an) <= 1e-3 * np.linalg.norm(fd), (fd, an)
        ent = rng.choice(tsel, size=64, replace=False)
        tfb = start.tf.reshape(-1)
        fd = np.array([fd_of(lambda x, e=e: p.with_tf_entry(int(e), x), float(tfb[e])) for e in ent])
        an = gtf[ent]
        assert np.linalg.norm(fd - an) <= 1e-3 * np.linalg.norm(fd), (fd, an)


def _march_both_ways(scene, views, step, store=None):
    """The march in one call, whose pixels call for the search of empty
    blocks, and view by view, which takes every step."""
    import torch
    both = EAProblem(scene, views, step, store=store).render()
    each = torch.cat([EAProblem(scene, [v], step, store=store).render() for v in views])
    torch.cuda.synchronize()
    return both.cpu().numpy(), each.cpu().numpy()


@pytest.mark.parametrize("dims", [(49, 49, 49), (65, 50, 57), (100, 64, 81)])
@pytest.mark.parametrize("fmt", [None, N.GBV_VOXEL_F32, N.GBV_VOXEL_F16, N.GBV_VOXEL_U8_SCALED])
@pytest.mark.parametrize("kind", ["two_peaks", "opaque", "nan_voxels", "inside", "far", "negative"])
def test_skipped_steps_change_nothing(cuda, dims, fmt, kind):
    """Empty space is skipped from 768 k pixels on: the image is the one that
    takes every step, bit for bit, at block edges (a last block of one cell, a
    clipped one), for rays along the faces, from inside the box and from far
    away, with voxels that are NaN, with no empty block at all, and with
    negative opacities."""
    from barney_gb300.device import GpuScene
    s = scenes.Scene(scalars=scenes.blob_volume(dims, 12, seed=8, noise=0.0), tf=scenes.tf_two_peaks(256),
                     base_density=20.0)
    views = scenes.fibonacci_views(4, 2.5, 8)
    if kind == "opaque":
        s.tf = scenes.tf_ramp(64) + np.float32(0.01)
    if kind == "nan_voxels":
        s.scalars[3, 5, 7] = np.nan
    if kind == "negative":
        s.tf[:, 3] *= -0.1
    for k, v in enumerate(views):
        v["width"], v["height"] = 640, 400
        if kind == "inside":
            v["pos"] = (0.1 * k, -0.05, 0.02)
        if kind == "far":
            v["pos"] = tuple(40.0 * x for x in v["pos"])
            v["fovy"] = 1.0
    views[0]["pos"], views[0]["dir"] = (0.0, 0.0, 2.0), (0.0, 0.0, -1.0)  # rays along the axes
    store = GpuScene(s, fmt=fmt) if fmt is not None else None
    both, each = _march_both_ways(s, views, 0.5 / (max(dims) - 1), store)
    np.testing.assert_array_equal(both.view(np.uint32), each.view(np.uint32))


@pytest.mark.parametrize("entry", [np.inf, np.nan, 1e38])
def test_transfer_functions_that_rule_skipping_out(cuda, entry):
    """An entry whose product with zero, or whose optical depth, is not finite."""
    s = scenes.Scene(scalars=scenes.blob_volume((64, 64, 64), 12, seed=8, noise=0.0), tf=scenes.tf_two_peaks(256),
                     base_density=20.0)
    s.tf[10, 3 if entry == 1e38 else 0] = entry
    views = scenes.fibonacci_views(4, 2.5, 8)
    for v in views:
        v["width"], v["height"] = 640, 400
    both, each = _march_both_ways(s, views, 0.5 / 63)
    np.testing.assert_array_equal(both.view(np.uint32), each.view(np.uint32))


@pytest.mark.parametrize("fmt", [None, N.GBV_VOXEL_F16])
def test_infinite_transmittance_is_not_skipped(cuda, fmt):
    """Opacities so negative that the transmittance overflows: a step of zero
    opacity past that point is 0 times infinity, in the march that looks for
    empty blocks as in the one that takes every step."""
    from barney_gb300.device import GpuScene
    s = scenes.Scene(scalars=scenes.blob_volume((64, 64, 64), 12, seed=8, noise=0.0), tf=scenes.tf_two_peaks(256),
                     base_density=20.0)
    s.tf[:, 3] *= -40.0
    views = scenes.fibonacci_views(4, 2.5, 8)
    for v in views:
        v["width"], v["height"] = 640, 400
    store = GpuScene(s, fmt=fmt) if fmt is not None else None
    both, each = _march_both_ways(s, views, 0.5 / 63, store)
    assert np.isnan(each).any()
    np.testing.assert_array_equal(both.view(np.uint32), each.view(np.uint32))


def test_adjoint_of_an_infinite_transmittance(cuda):
    """A slab of opacity -40 (30 steps of depth -13: the transmittance is
    infinite past it), then one of opacity 0: a step there has the weight
    infinity times 0, and so have the gradients of its transfer-function
    segment."""
    import torch
    n = 32
    s = scenes.Scene(scalars=np.full((n, 8, 8), 0.75, np.float32),
                     tf=np.ones((5, 4), np.float32), base_density=20.0)
    s.scalars[n // 2:] = 0.25  # the camera's side: entry 1 of 0..4; the far side: entry 3
    s.tf[:3, 3], s.tf[3:, 3] = -40.0, 0.0
    view = dict(scenes.fibonacci_views(1, 2.5, 8)[0], width=1, height=1, pos=(0.0, 0.0, 2.0), dir=(0.0, 0.0, -1.0),
                up=(0.0, 1.0, 0.0))
    p = EAProblem(s, [view], 0.5 / (n - 1))
    img = p.render()
    gv, gt = p.backward(img, torch.ones_like(img))
    torch.cuda.synchronize()
    assert np.isnan(img.cpu().numpy()[0, :3]).all()
    # the segment of entries 3 and 4 is met at opacity 0 alone
    assert np.isnan(gt.cpu().numpy()[3:]).all()


def _search_case():
    """A march of enough pixels to look for empty blocks, and gradients of its images."""
    import torch
    s = scenes.Scene(scalars=scenes.blob_volume((64, 64, 64), 12, seed=8, noise=0.0), tf=scenes.tf_two_peaks(256),
                     base_density=20.0)
    views = scenes.fibonacci_views(4, 2.5, 8)
    for v in views:
        v["width"], v["height"] = 640, 400
    p = EAProblem(s, views, 0.5 / 63)
    img = p.render()
    gimg = torch.rand(img.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    torch.cuda.synchronize()
    return p, img, gimg


class _Calls:
    """gbv_ea_render and gbv_ea_backward into buffers of their own, and what they are to hold."""

    def __init__(self, p, img, gimg):
        import torch
        self.p, self.img, self.gimg = p, img, gimg
        self.gv, self.gt = p.backward(img, gimg)
        self.out, self.cv, self.ct = torch.empty_like(img), torch.zeros_like(self.gv), torch.zeros_like(self.gt)
        self.rec = p.record()

    def clear(self):
        import torch
        for t in (self.out, self.cv, self.ct):
            t.zero_()
        torch.cuda.synchronize()

    def run(self, stream):
        import ctypes as C
        p, n = self.p, len(self.p.views)
        N.check(N.lib().gbv_ea_render(C.byref(self.rec), p._views_c, n, p.step, self.out.data_ptr(), stream))
        N.check(N.lib().gbv_ea_backward(C.byref(self.rec), p._views_c, n, p.step, self.img.data_ptr(),
                                        self.gimg.data_ptr(), self.cv.data_ptr(), self.ct.data_ptr(), stream))

    def check(self):
        import torch
        torch.cuda.synchronize()
        np.testing.assert_array_equal(self.out.cpu().numpy().view(np.uint32), self.img.cpu().numpy().view(np.uint32))
        # the gradients' additions may be in another order: each entry's
        # rounding is far below 1e-5 of the largest
        for got, ref in ((self.cv, self.gv), (self.ct, self.gt)):
            np.testing.assert_allclose(got.cpu(), ref.cpu(), rtol=1e-4, atol=1e-5 * float(ref.abs().max()))


def _runtime():
    import ctypes as C
    return C.CDLL(next(x.split()[-1] for x in open("/proc/self/maps") if "libcudart" in x))


@pytest.mark.parametrize("fmt", [None, N.GBV_VOXEL_F16])
def test_empty_blocks_are_looked_for(cuda, fmt):
    """The four views of the tests that compare the two marches call for the
    search, one of them alone does not."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    from barney_gb300.device import GpuScene
    p, _, _ = _search_case()
    store = GpuScene(p.s, fmt=fmt) if fmt is not None else None
    for views, searches in ((p.views, 1), (p.views[:1], 0)):
        q = EAProblem(p.s, views, p.step, store=store)
        for _ in range(2):  # a profiler's first session may record nothing
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                q.render()
                torch.cuda.synchronize()
            names = [e.name for e in prof.events() if "gbv::" in e.name]
        assert sum("ea_forward_kernel" in n for n in names) == 1
        assert sum("empty_kernel" in n or "empty_ranges_kernel" in n for n in names) == searches


def test_captured_march_and_adjoint(cuda):
    """A capture of the march and its adjoint holds kernels alone: the graph
    can be cloned, put into another one and instantiated twice, and each
    replay gives the calls' results."""
    import ctypes as C
    import torch
    rt, calls = _runtime(), _Calls(*_search_case())
    stream = torch.cuda.Stream()
    st = C.c_void_p(stream.cuda_stream)
    graph, clone, parent, node = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(st, 1) == 0
    calls.run(st)
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0
    assert rt.cudaGraphClone(C.byref(clone), graph) == 0
    assert rt.cudaGraphCreate(C.byref(parent), 0) == 0
    assert rt.cudaGraphAddChildGraphNode(C.byref(node), parent, None, C.c_size_t(0), graph) == 0
    for g in (graph, graph, clone, parent):
        exe = C.c_void_p()
        assert rt.cudaGraphInstantiate(C.byref(exe), g, C.c_ulonglong(0)) == 0
        calls.clear()
        assert rt.cudaGraphLaunch(exe, st) == 0
        calls.check()


def test_march_and_adjoint_beside_a_capture(cuda):
    """The calls on one stream while another one is captured, in the mode that
    forbids allocations: both go on."""
    import ctypes as C
    import torch
    rt, calls = _runtime(), _Calls(*_search_case())
    other, mine = torch.cuda.Stream(), torch.cuda.Stream()
    graph = C.c_void_p()
    calls.clear()
    assert rt.cudaStreamBeginCapture(C.c_void_p(other.cuda_stream), 0) == 0
    calls.run(C.c_void_p(mine.cuda_stream))
    assert rt.cudaStreamEndCapture(C.c_void_p(other.cuda_stream), C.byref(graph)) == 0
    calls.check()


@pytest.mark.parametrize("w,h,nviews", [(1, 1, 1), (9, 5, 3), (33, 17, 2), (16, 8, 33)])
def test_adjoint_tiles_of_uneven_views(cuda, w, h, nviews):
    """Views whose tiles are partial, and more of them than one launch holds:
    the gradients are the sums of the views' own (to the order of their
    additions: each entry's rounding is below the sum of its terms' sizes
    times the number of additions)."""
    gt = scenes.ea_scene(24)
    views = scenes.fibonacci_views(nviews, 2.5, 8)
    for k, v in enumerate(views):
        v["width"], v["height"] = w + k % 2, h
    step = 0.5 / 23
    p = EAProblem(gt, views, step)
    img = p.render()
    gv, gt_tf = p.backward(img, img)
    sv, st, at = 0.0, 0.0, 0
    for v in views:
        n = v["width"] * v["height"]
        part = img[at:at + n].contiguous()
        a, b = EAProblem(gt, [v], step).backward(part, part)
        sv, st, at = sv + a.double(), st + b.double(), at + n
    np.testing.assert_allclose(gv.double().cpu(), sv.cpu(), rtol=1e-4, atol=1e-5 * float(sv.abs().max()))
    np.testing.assert_allclose(gt_tf.double().cpu(), st.cpu(), rtol=1e-4, atol=1e-5 * float(st.abs().max()))
