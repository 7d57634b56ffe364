"""Device-built trees of meshes that are split level by level: edges of the
blocks that share a task, more levels than even halves need, coincident
centroids (halved by index) and many meshes at once; every closest hit equals
the host-built tree's bit for bit."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import _abi as A

pytestmark = pytest.mark.gpu


def _mesh(n, kind, rng):
    c = rng.uniform(-1, 1, (n, 3))
    if kind == "lopsided":  # a split takes off a twentieth of the primitives at a time
        c = np.sign(c) * 2.0 ** (-20.0 * rng.random((n, 1)) ** 0.5) * np.abs(c)
    elif kind == "together":
        c[:] = 0.1
    shape = rng.uniform(-0.02, 0.02, (n, 3, 3))
    if kind == "together":
        shape[:] = shape[0]
    v = np.zeros(3 * n, A.VERTEX_DTYPE)
    v["pos"] = (c[:, None] + shape).astype(np.float32).reshape(-1, 3)
    v["normal"] = (0, 0, 1)
    return v


@pytest.mark.parametrize("kind,sizes", [("spread", [513]), ("spread", [4096]), ("spread", [4097]), ("spread", [30011]),
                                        ("lopsided", [20000]), ("together", [9000]),
                                        ("spread", [1, 512, 513, 1025, 4095, 8193, 3, 700, 5000, 513])])
def test_large_meshes_equal_host_tree(ctx, kind, sizes):
    rng = np.random.default_rng(sum(sizes))
    b = ag.SceneBuilder()
    m = b.add_lambertian("m", (0.5, 0.5, 0.5))
    verts = [_mesh(n, kind, rng) for n in sizes]
    for k, v in enumerate(verts):
        b.add_mesh("t%d" % k, v, np.arange(len(v), dtype=np.uint32))
        b.add_instance("t%d" % k, m)
    d = b.desc()
    dev = ctx.create_scene(d)
    ctx.set_bvh_build(on_device=False)
    try:
        host = ctx.create_scene(d)
    finally:
        ctx.set_bvh_build(on_device=True)
    pos = np.concatenate([v["pos"].reshape(-1, 3, 3).mean(1) for v in verts])
    o = (rng.normal(size=(4000, 3)) * 2).astype(np.float32)
    dirs = (pos[rng.integers(0, len(pos), 4000)] - o).astype(np.float32)
    h1, i1 = dev.trace(o, dirs)
    h2, i2 = host.trace(o, dirs)
    assert np.array_equal(i1, i2) and np.array_equal(h1.view(np.uint32), h2.view(np.uint32))
    assert (i1 != 0xFFFFFFFF).sum() > 0
