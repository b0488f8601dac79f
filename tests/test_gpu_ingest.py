"""What makes a volume ready to render, at the edges of its kernels' tiles:
macrocell ranges by strips of columns, normalised texels by 16-byte vectors,
the env light's tables by warps, a NanoVDB grid's ranges by leaves.  All are
exact: numpy's min and max, IEEE division, the oracle's tables."""
import ctypes as C

import numpy as np
import pytest

from barney_gb300 import _native as N
from barney_gb300 import nanovdb, scenes
from barney_gb300.device import _ptr, _stream, mc_dims
import oracle

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def ranges_of(vol, first, last):
    """(min, max) over the windows [first, last] per axis (x, y, z lists), NaN
    never replacing a bound."""
    lo = np.where(np.isnan(vol), np.inf, vol)
    hi = np.where(np.isnan(vol), -np.inf, vol)
    for axis, dim in ((0, 2), (1, 1), (2, 0)):
        cut = [(a, b + 1) for a, b in zip(first[axis], last[axis])]
        lo = np.stack([lo.take(range(a, b), dim).min(dim) for a, b in cut], dim)
        hi = np.stack([hi.take(range(a, b), dim).max(dim) for a, b in cut], dim)
    return np.stack([lo, hi], -1).reshape(-1, 2).astype(np.float32)


@pytest.mark.parametrize("dims,cpm", [((2, 2, 2), 1), ((129, 3, 4), 1), ((130, 5, 9), 8), ((128, 17, 33), 16),
                                      ((129, 18, 16), 16), ((257, 34, 20), 16), ((140, 9, 7), 3), ((88, 45, 50), 43),
                                      ((131, 66, 70), 64), ((140, 70, 66), 65), ((300, 20, 30), 150),
                                      ((64, 64, 64), 128)])
def test_macrocell_ranges_at_strip_edges(cuda, dims, cpm):
    import torch
    rng = np.random.default_rng(3)
    nx, ny, nz = dims
    vol = rng.normal(size=(nz, ny, nx)).astype(np.float32)
    vol.flat[rng.integers(0, vol.size, 3)] = np.nan
    vol.flat[rng.integers(0, vol.size, 2)] = [np.inf, -np.inf]
    M = mc_dims(dims, cpm)
    d = torch.from_numpy(vol).cuda()
    out = torch.empty((M[0] * M[1] * M[2], 2), dtype=torch.float32, device="cuda")
    N.check(N.lib().gbv_build_mc_ranges(_ptr(d), N.ivec(*dims), cpm, _ptr(out), _stream()), "gbv_build_mc_ranges")
    want = ranges_of(vol, [[m * cpm for m in range(k)] for k in M],
                     [[min(n - 1, (m + 1) * cpm) for m in range(k)] for n, k in zip(dims, M)])
    np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(want))


@pytest.mark.parametrize("nx", [2, 3, 5, 9, 16, 17, 33, 63, 64])
@pytest.mark.parametrize("cpm", [1, 2, 3, 4, 8, 16, 31, 64, 200])
def test_macrocell_ranges_of_thin_fields(cuda, nx, cpm):
    """Fields of few voxels along x: blocks that hold several rows of
    macrocells, the last one fewer; slices of one row and of many."""
    test_macrocell_ranges_at_strip_edges(cuda, (nx, 43, 37), cpm)
    test_macrocell_ranges_at_strip_edges(cuda, (nx, 2, 67), cpm)


@pytest.mark.parametrize("bits_,shift", [(8, 0), (8, 3), (16, 0), (16, 2)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4096, 4099])
def test_normalized_texels_at_vector_edges(cuda, bits_, shift, n):
    """shift: bytes past a 16-byte boundary the texels start at."""
    import torch
    dt = np.uint8 if bits_ == 8 else np.uint16
    t = np.random.default_rng(n).integers(0, 2 ** bits_, n).astype(dt)
    raw = torch.zeros(n * t.itemsize + 32, dtype=torch.uint8, device="cuda")
    raw[shift:shift + n * t.itemsize] = torch.from_numpy(t.view(np.uint8)).cuda()
    out = torch.full((n + 4,), -1.0, device="cuda")
    N.check(N.lib().gbv_normalize_texels(C.c_void_p(raw.data_ptr() + shift), bits_, n, _ptr(out), _stream()),
            "gbv_normalize_texels")
    got = out.cpu().numpy()
    np.testing.assert_array_equal(bits(got[:n]), bits(t.astype(np.float32) / np.float32(2 ** bits_ - 1)))
    assert (got[n:] == -1.0).all()


@pytest.mark.parametrize("w,h", [(1, 1), (31, 33), (32, 5), (33, 100), (200, 31), (513, 64)])
@pytest.mark.parametrize("addr", [(N.GBV_ADDR_WRAP, N.GBV_ADDR_CLAMP), (N.GBV_ADDR_MIRROR, N.GBV_ADDR_WRAP)])
def test_env_tables_at_warp_edges(cuda, w, h, addr):
    import torch
    tex = np.random.default_rng(w * 1000 + h).uniform(0.0, 3.0, (h, w, 4)).astype(np.float32)
    d = torch.from_numpy(tex).cuda()
    cy, cx = torch.empty(h, device="cuda"), torch.empty(h * w, device="cuda")
    N.check(N.lib().gbv_env_build_cdfs(_ptr(d), w, h, N.ivec(*addr), _ptr(cy), _ptr(cx), _stream()),
            "gbv_env_build_cdfs")
    oy, ox = oracle.env_cdfs(tex, addr)
    np.testing.assert_array_equal(bits(cx.cpu().numpy()), bits(ox.reshape(-1)))
    # the device's bounded sine is within 2 ulp of libm's: each of the h terms
    # and each of the 2 h additions may round another way
    np.testing.assert_allclose(cy.cpu().numpy(), oy, rtol=(2 + 2 * h) * 2.0 ** -23)


@pytest.mark.parametrize("dims,origin", [((1, 1, 1), (0, 0, 0)), ((17, 16, 33), (0, 0, 0)), ((50, 21, 40), (-13, 5, -100)),
                                         ((9, 130, 20), (4090, -3, 7))])
@pytest.mark.parametrize("coarse", [False, True])
def test_nanovdb_ranges_at_leaf_edges(cuda, dims, origin, coarse):
    """Leaves, missing leaves (background) and root tiles across 4096; coarse:
    a caller's own macrocells, larger than the parsed ones."""
    import torch
    rng = np.random.default_rng(7)
    nx, ny, nz = dims
    vol = rng.uniform(0.1, 1.0, (nz, ny, nx)).astype(np.float32)
    vol[rng.random(vol.shape) < 0.02] = 0.0
    if min(dims) > 16:
        vol[:, :, 8:16] = 0.0
    vol[0, 0, 0] = vol[-1, -1, -1] = 0.5  # the index box is the array's
    g = scenes.nanovdb_grid(vol, origin, 1.0, background=0.0)
    info = nanovdb.parse(g)
    lo = np.array(list(info.index_lo))
    size = np.array(list(info.index_hi)) - lo + 1
    if coarse:
        info.mc_dims[:] = [max(1, int(m) // 3) for m in info.mc_dims]
    mc = list(info.mc_dims)
    d = torch.from_numpy(np.frombuffer(g, np.uint8).copy()).cuda()
    out = torch.empty((mc[0] * mc[1] * mc[2], 2), dtype=torch.float32, device="cuda")
    N.check(nanovdb.lib().gbv_nanovdb_mc_ranges(_ptr(d), C.byref(info), _ptr(out), _stream()),
            "gbv_nanovdb_mc_ranges")
    # the grid's own values, as the sampler reads them at voxel centres
    pad = size + 2
    k, j, i = np.meshgrid(*[np.arange(n) for n in pad[::-1]], indexing="ij")
    values = np.zeros(pad[::-1], np.float32)
    inside = (i < size[0]) & (j < size[1]) & (k < size[2])
    pts = np.stack([i[inside] + lo[0], j[inside] + lo[1], k[inside] + lo[2]], -1).astype(np.float32) + np.float32(0.5)
    p = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    v = torch.empty(len(pts), device="cuda")
    N.check(nanovdb.lib().gbv_nanovdb_sample(_ptr(d), C.byref(info), _ptr(p), len(pts), _ptr(v), _stream()),
            "gbv_nanovdb_sample")
    values[inside] = v.cpu().numpy()
    want = ranges_of(values, [[m * s // c for m in range(c)] for s, c in zip(size, mc)],
                     [[(m + 1) * s // c + 1 for m in range(c)] for s, c in zip(size, mc)])
    np.testing.assert_array_equal(bits(out.cpu().numpy()), bits(want))
