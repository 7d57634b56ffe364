"""Device-built bottom-level trees around the sizes of the one-warp sweep (32
primitives, and the subtrees handed to a warp): every closest hit equals the
host-built tree's bit for bit, with spread, coincident and collinear
centroids.  The hits depend on the triangles alone, so the tolerance is zero."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import _abi as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spread", "together", "line", "two_places"])
@pytest.mark.parametrize("n", [2, 6, 31, 32, 33, 63, 64, 65, 511, 512, 513, 1500])
def test_device_tree_equals_host_tree(ctx, n, kind):
    rng = np.random.default_rng(n)
    c = rng.uniform(-1, 1, (n, 3))
    if kind == "together":
        c[:] = 0.1
    elif kind == "line":
        c[:, 1:] = 0.25
    elif kind == "two_places":
        c = np.where(rng.random((n, 1)) < 0.5, -0.5, 0.5) * np.ones(3)
    shape = rng.uniform(-0.1, 0.1, (n, 3, 3)) if kind in ("spread", "line") else \
        np.tile(rng.uniform(-0.1, 0.1, (1, 3, 3)), (n, 1, 1))
    v = np.zeros(3 * n, A.VERTEX_DTYPE)
    v["pos"] = (c[:, None] + shape).astype(np.float32).reshape(-1, 3)
    v["normal"] = (0, 0, 1)
    b = ag.SceneBuilder()
    m = b.add_lambertian("m", (0.5, 0.5, 0.5))
    b.add_mesh("t", v, np.arange(3 * n, dtype=np.uint32))
    b.add_instance("t", m)
    d = b.desc()
    dev = ctx.create_scene(d)
    ctx.set_bvh_build(on_device=False)
    try:
        host = ctx.create_scene(d)
    finally:
        ctx.set_bvh_build(on_device=True)
    o = (rng.normal(size=(2000, 3)) * 2).astype(np.float32)
    dirs = (v["pos"].reshape(-1, 3, 3).mean(1)[rng.integers(0, n, 2000)] - o).astype(np.float32)
    h1, i1 = dev.trace(o, dirs)
    h2, i2 = host.trace(o, dirs)
    assert np.array_equal(i1, i2) and np.array_equal(h1.view(np.uint32), h2.view(np.uint32))
    assert (i1 != 0xFFFFFFFF).sum() > 0
