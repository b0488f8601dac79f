"""The library's scratch memory: its pool's errors and captures against a fake
CUDA runtime (CPU), and that what it keeps is given back (GPU)."""
import subprocess
from pathlib import Path

import pytest

from barney_gb300 import _native as N
from barney_gb300 import bn, scenes

ROOT = Path(__file__).resolve().parent.parent


def test_pool_against_a_fake_runtime(tmp_path):
    exe = tmp_path / "scratch_check"
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(ROOT / "tests" / "c" / "fake_cuda"),
                        str(ROOT / "tests" / "c" / "scratch_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert (r.returncode, r.stdout) == (0, "ok\n")


@pytest.mark.gpu
@pytest.mark.parametrize("by", ["call", "context"])
def test_kept_scratch_is_given_back(cuda, by):
    """A frame with a log of some 490 MB: the library keeps it, until it is
    asked for it or the device's last context goes."""
    import torch
    from barney_gb300.device import GpuScene
    s = scenes.small_scene(dims=40, spp=1, width=640, height=400)
    s.cam_pos = (0.05, 0.02, 0.03)  # inside: every tile sees the field
    g = GpuScene(s)
    acc = g.new_accum()
    session = bn.BarneySession() if by == "context" else None
    g.render(spp=90, accum=acc)
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    if by == "call":
        N.check(N.lib().gbv_release_scratch(), "gbv_release_scratch")
    else:
        session.close()
    assert torch.cuda.mem_get_info()[0] - kept >= 400 << 20
    g.render(spp=90, accum=acc)  # and takes it again
    torch.cuda.synchronize()
    N.check(N.lib().gbv_release_scratch(), "gbv_release_scratch")
