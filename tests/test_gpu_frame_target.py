"""The memory a frame is drawn into: stored by the shading pass, copied, or refused."""

import ctypes as C

import numpy as np
import pytest
import torch

from harness import build_gpu, gaussian_pair
from isaac_b200 import _lib, scenes

pytestmark = pytest.mark.gpu

FB = (61, 37)  # no multiple of a tile
BYTES = 4 * FB[0] * FB[1]
SENTINEL = 171


def _render(viz, ptr):
    _lib.check(viz.lib.isaacb_render(viz.ctx, viz._stream(), C.c_void_p(ptr)), viz.ctx)
    torch.cuda.synchronize()


@pytest.mark.parametrize("target", ["device", "device+1", "device+2", "device+4", "pinned", "pinned+1"])
def test_frame_reaches_the_target(target):
    viz = build_gpu(gaussian_pair(32, fb=FB))
    ref = viz.doVisualization().reshape(-1)
    kind, _, off = target.partition("+")
    off = int(off or 0)
    buf = torch.full((BYTES + 16,), SENTINEL, dtype=torch.uint8, device="cuda" if kind == "device" else "cpu")
    if kind == "pinned":
        buf = buf.pin_memory()
    _render(viz, buf.data_ptr() + off)
    got = buf.cpu().numpy()
    assert np.array_equal(got[off : off + BYTES], ref)
    assert (got[:off] == SENTINEL).all() and (got[off + BYTES :] == SENTINEL).all()
    viz.close()


def test_frame_into_the_framebuffer_itself():
    viz = build_gpu(gaussian_pair(32, fb=FB))
    ref = viz.doVisualization()
    own = C.c_void_p()
    _lib.check(viz.lib.isaacb_framebuffer(viz.ctx, C.byref(own)), viz.ctx)
    viz.setRenderMode(3)
    viz.render()
    viz.setRenderMode(0)
    _render(viz, own.value)
    out = torch.empty((FB[1], FB[0], 4), dtype=torch.uint8, device="cuda")
    viz.render(out)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)
    viz.close()


def test_pageable_memory_is_refused_before_any_launch():
    viz = build_gpu(gaussian_pair(32, fb=FB))
    ref = viz.doVisualization()
    out = torch.full((FB[1], FB[0], 4), SENTINEL, dtype=torch.uint8)
    for call in (lambda: viz.render(out), lambda: viz.doVisualization(host=False, out=out)):
        with pytest.raises(_lib.IsaacError) as e:
            call()
        assert e.value.status == _lib.INVALID_ARG
    torch.cuda.synchronize()
    assert (out == SENTINEL).all()
    assert np.array_equal(viz.doVisualization(), ref)
    viz.close()


@pytest.mark.parametrize("fb", [(61, 37), (256, 256), (257, 256)])
def test_host_frames_pageable_and_pinned(fb):
    """Frames that pass the context's own pinned buffer, the largest of them and the next
    size, into memory of either kind, twice each, with one camera and then another."""
    viz = build_gpu(gaussian_pair(32, fb=fb))
    dev = torch.empty((fb[1], fb[0], 4), dtype=torch.uint8, device="cuda")
    pageable = np.full((fb[1], fb[0], 4), SENTINEL, dtype=np.uint8)
    pinned = torch.full((fb[1], fb[0], 4), SENTINEL, dtype=torch.uint8).pin_memory().numpy()
    seen = []
    for seed in (1, 7):
        viz.setCamera(*scenes.camera(*fb, seed=seed))
        ref = viz.doVisualization(host=False, out=dev).cpu().numpy()
        for out in (pageable, pinned, pageable):
            assert viz.doVisualization(out=out) is out
            assert np.array_equal(out, ref)
        seen.append(ref)
    assert not np.array_equal(*seen)
    viz.close()
