"""The memory a frame is drawn into: stored by the shading pass, copied, or refused."""

import ctypes as C

import numpy as np
import pytest
import torch

from harness import assert_image_parity, build_gpu, build_oracle, gaussian_pair
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


def _pass_scene(kind):
    """Scenes for every kernel that can end a frame, with every choice of the passes before
    it."""
    per_source = kind.startswith("per_source")
    s = gaussian_pair(24, fb=FB, background=(0.2, 0.4, 0.6, 1.0), optimized=not per_source)
    scalar = s.volumes[0][0]
    if per_source and "vector" not in kind:
        count = {"one": 1, "two": 2, "three": 3, "five": 5}[kind.split("_")[2]]
        s.volumes = [(np.roll(scalar, 3 * i, axis=0).copy(), True) for i in range(count)]
        s.functions, s.transfer = ["idem"] * count, [scenes.transfer_4point(0.4 * i) for i in range(count)]
    n = len(s.volumes)
    s.interpolation = "nearest" not in kind
    s.weights = [0.0] * n if "weightless" in kind else [2.0] * n
    if "iso" in kind:
        s.iso = [0.4] + [0.0] * (n - 1)
    if "ssao" in kind:
        s.ao = (True, 0.7, False)
    if "particles" in kind:
        off, pos, attr = scenes.particles_uniform(400, (8, 8, 8), seed=5)
        s.particle_cells = (8, 8, 8)
        s.particles = [(off.numpy(), pos.numpy(), attr.numpy(), None, 0.5)]
        s.functions = s.functions + ["length"]
        s.transfer = s.transfer + [{0: (0.1, 0.9, 0.1, 1.0), 1024: (0.9, 0.1, 0.1, 1.0)}]
        s.weights = s.weights + [2.0]
    return s


@pytest.mark.parametrize("mode", [0, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("kind", [
    "combined", "combined_nearest", "combined_weightless", "combined_iso", "combined_iso_ssao", "combined_ssao",
    "combined_particles", "combined_particles_iso_ssao", "per_source_one", "per_source_two_nearest", "per_source_three",
    "per_source_three_ssao", "per_source_two_iso", "per_source_two_particles", "per_source_five", "per_source_vector",
    "per_source_vector_iso", "per_source_one_weightless"])
def test_every_pass_stores_the_frame_and_the_buffers(kind, mode):
    """The frame stored into the caller's memory is the framebuffer's on every pixel, and the
    frame, depth and occlusion are the oracle's whichever pass cleared them."""
    s = _pass_scene(kind)
    s.render_mode = mode
    oracle = build_oracle(s)
    ref = oracle.frame()
    viz = build_gpu(s)
    host = viz.doVisualization()
    assert_image_parity(host, ref)
    rd, _, rao = oracle.gbuffer()
    for fill in (SENTINEL, 0):  # a second frame starts from the first one's buffers
        out = torch.full((FB[1], FB[0], 4), fill, dtype=torch.uint8, device="cuda")
        viz.doVisualization(host=False, out=out)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), host)
        gd, _, gao = viz.gbuffer()
        clear = rd > 1e30
        assert np.array_equal(gd[clear], rd[clear])
        assert np.allclose(gd[~clear], rd[~clear], rtol=1e-4, atol=1e-4)
        assert np.array_equal(gao, rao)
    viz.close()
