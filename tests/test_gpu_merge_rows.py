"""The merge of sources of any kind (functor chains, vectors, ghost cells, iso output,
rows of any length) and the vectorised min/max at the sizes where their groups, tails and
table limits can go wrong: textures and min/max bit-exact against the oracle."""

import numpy as np
import pytest
import torch

from harness import Scene, build_gpu, build_oracle
from isaac_b200 import scenes

pytestmark = pytest.mark.gpu

CHAINS = {1: ["idem", "mul(1.5)|add(-0.1)", "add(0.25)|length", "sum|mul(0.5)"],
          2: ["length", "mul(0.5,2)|sum"], 3: ["length", "sum|mul(0.4)", "idem"], 4: ["length|add(0.1)", "mul(1,2,3,4)|length"]}


def _scene(size, fdims, seed, guard=0, **kw):
    x, y, z = size
    rng = np.random.default_rng(seed)
    vols, functions = [], []
    for i, fd in enumerate(fdims):
        a = rng.uniform(-0.2, 1.0, (z, y, x) if fd == 1 else (z, y, x, fd)).astype(np.float32)
        if guard:
            full = rng.uniform(-50.0, 50.0, tuple(n + 2 * guard for n in a.shape[:3]) + a.shape[3:]).astype(np.float32)
            full[guard:-guard, guard:-guard, guard:-guard] = a
            a = full
        vols.append((a, True))
        functions.append(CHAINS[fd][(seed + i) % len(CHAINS[fd])])
    s = Scene(n=size, volumes=vols, functions=functions, guard=[guard] * len(vols))
    s.transfer = [scenes.transfer_4point(0.7 * i) for i in range(len(vols))]
    for k, v in kw.items():
        setattr(s, k, v)
    return s


def _check(s):
    o = build_oracle(s)
    o.update()
    rv, ri = o.combined()
    viz = build_gpu(s)
    viz.update()
    gv, gi = viz.combinedTextures()
    assert np.array_equal(gv, rv)
    assert np.array_equal(gi, ri)
    rmn, rmx = o.minmax()
    gmn, gmx = viz.minMax()
    assert rmn.tobytes() == gmn.tobytes() and rmx.tobytes() == gmx.tobytes()
    viz.close()


@pytest.mark.parametrize("size", [(1, 1, 1), (1, 7, 5), (31, 3, 2), (33, 1, 65), (64, 9, 1), (130, 17, 3)])
@pytest.mark.parametrize("fdims", [(1,), (1, 3), (4, 1, 2), (1, 1, 1, 1), (3, 1, 1, 3, 1)])
def test_sizes_and_source_counts(size, fdims):
    """Fewer voxels than a warp, tails, rows of 1; 5 sources take the one-voxel kernel."""
    _check(_scene(size, fdims, seed=sum(size) + len(fdims)))


@pytest.mark.parametrize("dither", [0, 1, 2, 3, 5])
@pytest.mark.parametrize("guard", [0, 2])
@pytest.mark.parametrize("weights", [(2.0, 1.0, 0.25), (0.5, 0.0, 1.5), (1.0, -0.5, 2.0), (1e-8, 0.0, 0.0), (3e6, 1.0, 1.0)])
def test_weights_iso_guard_and_dither(dither, guard, weights):
    """Total weights that are and are not powers of two, negative, and beyond what the
    reciprocal division takes; iso thresholds on weighted and unweighted sources."""
    _check(_scene((37, 21, 10), (1, 3, 1), seed=dither, guard=guard, weights=list(weights), iso=[0.0, 0.45, 0.3], dither_mode=dither))


@pytest.mark.parametrize("ts", [2, 100, 2048, 8192])
def test_transfer_sizes(ts):
    """Tables that fit in shared memory, for one or all sources, and that do not."""
    s = _scene((40, 12, 9), (3, 1, 1), seed=3, transfer_size=ts, iso=[0.4, 0.0, 0.0])
    s.transfer = [{0: (0.1, 0.2, 0.3, 0.0), ts // 2: (0.9, 0.4, 0.1, 0.6), ts: (0.2, 0.8, 0.9, 0.9)}] * 3
    _check(s)


def test_special_values():
    """NaN, infinities, signed zeros and subnormals in sources and tables."""
    s = _scene((33, 8, 6), (1, 3), seed=5)
    a, b = s.volumes[0][0], s.volumes[1][0]
    a.reshape(-1)[:9] = [np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-40, -1e-40, 3e38, -3e38]
    b.reshape(-1)[40:46] = [np.nan, np.inf, -np.inf, -0.0, 1e-42, 3e38]
    s.transfer[0] = {0: (1e-30, 1e-38, 1e-20, 1e-12), 512: (3e38, 1.0, 2.0, 1.0), 1024: (0.0, 1e-45, 1.0, 1.0)}
    _check(s)


@pytest.mark.parametrize("offset", [0, 1])
def test_minmax_off_a_16_byte_boundary(offset):
    from isaac_b200 import IsaacVisualization, VolumeSource

    g = torch.Generator(device="cuda").manual_seed(2)
    buf = torch.randn(4 + 3 * 21 * 13 * 11, generator=g, device="cuda")
    t = buf[offset : offset + 3 * 21 * 13 * 11].view(11, 13, 21, 3)
    viz = IsaacVisualization("m", (16, 16), (21, 13, 11), (21, 13, 11), (1, 1, 1), (0, 0, 0), [VolumeSource("a", t)])
    viz.functions = ["idem"]
    viz.updateFunctions()
    mn, mx = viz.minMax()
    assert mn[0] == t[..., 0].min().item() and mx[0] == t[..., 0].max().item()
    viz.close()


@pytest.mark.parametrize("size", [(1, 5, 3), (37, 9, 4), (260, 3, 2), (40, 6, 5)])
@pytest.mark.parametrize("count", [1, 2, 3, 4])
@pytest.mark.parametrize("guard", [0, 1])
def test_scalar_sources_with_tables_beyond_shared_memory(size, count, guard):
    """Ragged and aligned rows, with ghost cells or none, with and without iso output."""
    ts = 8192
    for iso in ([], [0.0] * (count - 1) + [0.4]):
        s = _scene(size, (1,) * count, seed=sum(size) + count, guard=guard, transfer_size=ts, iso=iso)
        s.functions = ["idem"] * count
        s.transfer = [{0: (0.1, 0.2, 0.3, 0.0), ts // 2: (0.9, 0.4, 0.1, 0.6), ts: (0.2, 0.8, 0.9, 0.9)}] * count
        _check(s)
