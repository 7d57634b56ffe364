"""The 8-wide traversal nodes at the sizes where they can go wrong: meshes
around a node's eight children and a leaf's three triangles, boxes that
quantise badly (flat, far from the origin, of very different extents), rays
along the axes, and wavefronts far smaller than the grid.  Every closest hit
is compared with the oracle's own tree bit for bit: the hits depend on the
triangle test alone, so the tolerance is zero."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import _abi as A
from asuna_gb300 import scenes
from oracle import oracle_py

pytestmark = pytest.mark.gpu


def _scene(tris, transforms):
    b = ag.SceneBuilder()
    m = b.add_lambertian("m", (0.5, 0.5, 0.5))
    v = np.zeros(3 * len(tris), A.VERTEX_DTYPE)
    v["pos"] = np.asarray(tris, np.float32).reshape(-1, 3)
    v["normal"] = (0, 0, 1)
    b.add_mesh("t", v, np.arange(3 * len(tris), dtype=np.uint32))
    for t in transforms:
        b.add_instance("t", m, t)
    return b.desc(), v["pos"].reshape(-1, 3, 3).astype(np.float64)


def _compare(ctx, desc, o, d, tmin=1e-5):
    hits, inst = ctx.create_scene(desc).trace(o, d, tmin=tmin)
    ref = oracle_py.OracleScene(desc)
    found = 0
    for k in range(len(o)):
        r = ref.trace(o[k], d[k], tmin, 1e10)
        if r is None:
            assert inst[k] == 0xFFFFFFFF, k
            continue
        t, ii, prim, u, v = r
        got = (hits[k, 0], inst[k], hits[k, 3].view(np.uint32), hits[k, 1], hits[k, 2])
        assert got == (np.float32(t), ii, prim, np.float32(u), np.float32(v)), (k, got, r)
        found += 1
    return found


EYE = np.eye(3, 4, dtype=np.float32)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 9, 23, 24, 25, 65, 200])
def test_children_and_leaf_counts(ctx, n):
    rng = np.random.default_rng(n)
    c = rng.uniform(-1, 1, (n, 1, 3))
    tris = c + rng.uniform(-0.2, 0.2, (n, 3, 3))
    desc, pos = _scene(tris, [EYE])
    target = pos[rng.integers(0, n, 300)].mean(1) + rng.normal(size=(300, 3)) * 0.02
    o = (rng.normal(size=(300, 3)) * 2).astype(np.float32)
    d = (target - o).astype(np.float32)
    assert _compare(ctx, desc, o, d) > 100


@pytest.mark.parametrize("scale,offset", [((1, 1, 1), (0, 0, 0)), ((1, 1, 0), (0, 0, 0)), ((1, 0, 0.001), (3, 5, -2)),
                                          ((1e-3, 1e-3, 1e-3), (1000, -2000, 500)), ((1e4, 1e-2, 1), (0, 100, 0)),
                                          ((1e-6, 1e-6, 1e-6), (0, 0, 0))])
def test_boxes_that_quantise_badly(ctx, scale, offset):
    rng = np.random.default_rng(7)
    n = 400
    tris = (rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.1, 0.1, (n, 3, 3))) * scale + offset
    move = EYE.copy()
    move[:, 3] = np.array(scale, np.float32) * 2.5 + np.float32(1e-3)
    turned = scenes.rot_y(33.0, -np.asarray(offset, np.float64) * 0.5)
    desc, pos = _scene(tris, [EYE, move, turned])
    target = pos[rng.integers(0, n, 400)].mean(1)
    size = max(np.abs(scale))
    o = (target + rng.normal(size=(400, 3)) * size).astype(np.float32)
    d = (target - o).astype(np.float32)
    # and along the axes, both ways, from a box's own planes
    o[:60] = (pos[:20].min(1)[:, None] - np.eye(3)[None] * size * 2).reshape(-1, 3)
    d[:60] = np.tile(np.eye(3), (20, 1))
    o[60:120] = (pos[:20].max(1)[:, None] + np.eye(3)[None] * size * 2).reshape(-1, 3)
    d[60:120] = -np.tile(np.eye(3), (20, 1))
    assert _compare(ctx, desc, o, d, tmin=0.0) > 0


def test_many_instances_of_different_scales(ctx):
    rng = np.random.default_rng(3)
    tris = rng.uniform(-1, 1, (30, 1, 3)) + rng.uniform(-0.3, 0.3, (30, 3, 3))
    ts = []
    for k in range(100):
        t = scenes.rot_y(float(rng.uniform(0, 360)), rng.uniform(-10, 10, 3))
        t[:, :3] *= np.float32(10.0 ** rng.uniform(-2, 0.5))
        ts.append(t)
    desc, _ = _scene(tris, ts)
    o = rng.uniform(-12, 12, (600, 3)).astype(np.float32)
    d = (np.array([t[:, 3] for t in ts])[rng.integers(0, 100, 600)] - o).astype(np.float32)
    assert _compare(ctx, desc, o, d) > 0  # (not a vacuous comparison)


@pytest.mark.parametrize("width,height", [(1, 1), (5, 1), (33, 3), (97, 61)])
def test_wavefronts_smaller_than_the_grid(ctx, width, height):
    b, shot = scenes.plugin_scene(width, height, frames=2, max_depth=5, channels=("albedo", "normal", "depth"))
    desc = b.desc()
    film = ctx.create_film(width, height)
    ctx.render(ctx.create_scene(desc), shot, film)
    want, _, _ = oracle_py.OracleScene(desc).render(shot)
    # the bound of the other comparisons of films with the oracle
    assert np.all(np.abs(film.read(0) - want[0]) <= 1e-4 * np.abs(want[0]) + 1e-6)
