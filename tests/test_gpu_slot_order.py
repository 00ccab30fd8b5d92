"""The slot order that a texture in memory has (Geom::yfast) against the order of the next
merge: a draw takes the former, whatever has been captured, has failed or is asked for in
the meantime.  Frames are the same bytes in both orders."""

import math

import numpy as np
import pytest
import torch

from harness import build_gpu, gaussian_pair
from isaac_b200 import _lib, scenes
from isaac_b200.batch import IsaacBatch

pytestmark = pytest.mark.gpu

FB = (64, 48)
FRONT = scenes.orbit_camera(*FB, yaw=0.0, pitch=0.6)  # merged x fastest by a context
SIDE = scenes.orbit_camera(*FB, yaw=math.pi / 2, pitch=0.1)  # y fastest


def _viz(seed=1, camera=FRONT):
    return build_gpu(gaussian_pair(32, fb=FB, seed=seed, P=camera[0], MV=camera[1]))


def _frame(viz):
    out = torch.zeros((FB[1], FB[0], 4), dtype=torch.uint8, device="cuda")
    viz.render(out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _reference(seed=1, camera=FRONT):
    viz = _viz(seed, camera)
    frame = viz.doVisualization()
    viz.close()
    assert frame.any()
    return frame


def test_draws_between_capture_and_launch():
    """A capture merges nothing: the context and the batch draw the texture as it is."""
    viz = _viz()
    batch = IsaacBatch([viz], [(0, *FB, *SIDE)])
    front, side = _reference(), _reference(camera=SIDE)
    viz.update()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        batch.capture(update=True)
    stream.synchronize()
    assert np.array_equal(_frame(viz), front)
    batch.render(update=False)
    torch.cuda.synchronize()
    assert np.array_equal(batch.frames[0].cpu().numpy(), side)
    for _ in range(2):
        batch.frames[0].zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            batch.launchGraph()
        stream.synchronize()
        assert np.array_equal(batch.frames[0].cpu().numpy(), side)
        assert np.array_equal(_frame(viz), front)
        viz.update()  # back to the context's own order
        assert np.array_equal(_frame(viz), front)
    batch.close()
    viz.close()


@pytest.mark.parametrize("how", ["render", "launchGraph"])
def test_draws_after_a_failed_update(how):
    """A batch update that stops at a context without memory leaves that context's texture,
    and every draw of either context is right afterwards."""
    vis = [_viz(1), _viz(2)]
    refs = [_reference(1), _reference(2)]
    batch = IsaacBatch(vis, [(0, *FB, *SIDE), (1, *FB, *SIDE)])
    stream = torch.cuda.Stream()
    for v in vis:
        v.update()
    torch.cuda.synchronize()
    if how == "launchGraph":
        with torch.cuda.stream(stream):
            batch.capture(update=True)
        stream.synchronize()
    keep = vis[1].volumeSources[0].data.data_ptr()
    _lib.check(vis[1].lib.isaacb_set_source(vis[1].ctx, 0, None), vis[1].ctx)
    with torch.cuda.stream(stream):
        with pytest.raises(_lib.IsaacError) as e:
            batch.render(update=True) if how == "render" else batch.launchGraph()
    assert e.value.status == _lib.NOT_READY
    stream.synchronize()
    for v, ref in zip(vis, refs):
        assert np.array_equal(_frame(v), ref)
    batch.render(update=False)
    torch.cuda.synchronize()
    for i in range(2):
        assert np.array_equal(batch.frames[i].cpu().numpy(), _reference(i + 1, SIDE))
    _lib.check(vis[1].lib.isaacb_set_source(vis[1].ctx, 0, keep), vis[1].ctx)
    batch.close()
    for v in vis:
        v.close()


def test_slot_order_setting_reaches_a_captured_graph():
    """setSlotOrder after a capture takes effect with the next launch, and the draws that
    follow read the texture in its new order."""
    viz = _viz()
    batch = IsaacBatch([viz], [(0, *FB, *SIDE)])
    front, side = _reference(), _reference(camera=SIDE)
    stream = torch.cuda.Stream()
    viz.update()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        batch.capture(update=True)
    for order in (0, 1, -1):
        viz.setSlotOrder(order)
        with torch.cuda.stream(stream):
            batch.launchGraph()
        stream.synchronize()
        assert np.array_equal(batch.frames[0].cpu().numpy(), side)
        assert np.array_equal(_frame(viz), front)
    batch.close()
    viz.close()


def test_update_captured_by_the_caller():
    """A caller's own graph holds an update: capturing it merges nothing, and after a replay
    or an update outside the graph, whatever the camera, every draw reads the right order."""
    viz = _viz()
    front, side = _reference(), _reference(camera=SIDE)
    out = torch.zeros((FB[1], FB[0], 4), dtype=torch.uint8, device="cuda")
    viz.update()
    assert np.array_equal(_frame(viz), front)
    viz.setCamera(*SIDE)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        viz.update()
        viz.render(out)
    assert np.array_equal(_frame(viz), side)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), side)
    for camera, want in ((FRONT, front), (SIDE, side)):
        viz.setCamera(*camera)
        viz.update()
        assert np.array_equal(_frame(viz), want)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), side)
        assert np.array_equal(_frame(viz), want)
    viz.close()


@pytest.mark.parametrize("interpolation", [True, False])
@pytest.mark.parametrize("fb", [(101, 77), (37, 29), (8, 3)])
@pytest.mark.parametrize("yaw,pitch", [(0.3, 0.2), (1.5, 0.5), (1.5, 0.6), (0.8, 1.0), (1.5, 1.5)])
def test_lanes_along_rows_and_down_columns(yaw, pitch, fb, interpolation):
    """Both lane orders of y-fastest slots (flat and steep cameras, pixels denser and wider
    than the voxels, ragged sizes) give the frame of x-fastest slots; batches too."""
    P, MV = scenes.orbit_camera(*fb, yaw=yaw, pitch=pitch)
    viz = build_gpu(gaussian_pair(32, fb=fb, P=P, MV=MV, interpolation=interpolation))
    batch = IsaacBatch([viz], [(0, *fb, P, MV)])
    frames = []
    for order in (0, 1):
        viz.setSlotOrder(order)
        frames.append(viz.doVisualization())
        batch.render(update=False)
        torch.cuda.synchronize()
        frames.append(batch.frames[0].cpu().numpy())
    assert frames[0].any()
    for f in frames[1:]:
        assert np.array_equal(f, frames[0])
    batch.close()
    viz.close()


def test_batch_orders_by_its_views():
    """One context under views from the front and the side, listed once or twice, single and
    captured, while cameras move: frames equal single views whatever order is chosen."""
    viz = _viz()
    front, side = _reference(), _reference(camera=SIDE)
    for ctxs, views in (([viz], [(0, *FB, *FRONT)] * 3 + [(0, *FB, *SIDE)]), ([viz, viz], [(0, *FB, *FRONT), (1, *FB, *SIDE), (1, *FB, *SIDE)])):
        batch = IsaacBatch(ctxs, views)
        want = [front if v[3] is FRONT[0] and v[4] is FRONT[1] else side for v in views]

        def check():
            torch.cuda.synchronize()
            for f, w in zip(batch.frames, want):
                assert np.array_equal(f.cpu().numpy(), w)
                f.zero_()
            assert np.array_equal(_frame(viz), front)

        batch.render(update=True)
        check()
        viz.update()
        batch.render(update=False)
        check()
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            batch.capture(update=True)
            batch.launchGraph()
        stream.synchronize()
        check()
        for i in range(len(views)):  # every view to the other side
            batch.setCamera(i, *(SIDE if want[i] is front else FRONT))
            want[i] = side if want[i] is front else front
        with torch.cuda.stream(stream):
            batch.launchGraph()
        stream.synchronize()
        check()
        batch.render(update=True)
        check()
        batch.close()
    viz.close()


def test_batch_over_a_context_whose_update_was_captured():
    """A batch merges in the order that the caller's graph writes, also where its own graph was
    captured before: after either one's merge every draw is right."""
    viz = _viz()
    front, side = _reference(), _reference(camera=SIDE)
    batch = IsaacBatch([viz], [(0, *FB, *SIDE)])
    viz.update()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        batch.capture(update=True)
        batch.launchGraph()  # y fastest, by its view
    stream.synchronize()
    viz.update()  # x fastest, by the camera
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        viz.update()
    for merge in (graph.replay, lambda: batch.render(update=True), graph.replay, batch.launchGraph, graph.replay, viz.update, graph.replay):
        with torch.cuda.stream(stream):
            merge()
        stream.synchronize()
        assert np.array_equal(_frame(viz), front)
        batch.frames[0].zero_()
        batch.render(update=False)
        torch.cuda.synchronize()
        assert np.array_equal(batch.frames[0].cpu().numpy(), side)
    batch.close()
    viz.close()
