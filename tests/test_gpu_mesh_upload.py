"""Meshes packed on the device: small, large and empty meshes in every order
(gathered and direct copies), triangle counts around the packing threshold
and around a block, and an index out of range.  Renders are compared with the
oracle (positions, normals, uvs and indices all show in the film's channels)
within the bound of the other film comparisons."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import _abi as A
from asuna_gb300 import scenes
from oracle import oracle_py

pytestmark = pytest.mark.gpu


def _patch(rng, n):
    """n triangles of a jittered grid in the unit square."""
    side = max(1, int(np.ceil(np.sqrt(n / 2))))
    g = np.stack(np.meshgrid(*[np.linspace(0, 1, side + 1)] * 2, indexing="ij"), -1).reshape(-1, 2)
    v = np.zeros(len(g), A.VERTEX_DTYPE)
    v["pos"][:, :2] = g
    v["pos"][:, 2] = rng.uniform(-0.05, 0.05, len(g))
    nrm = np.array([0, 0, 1]) + rng.uniform(-0.2, 0.2, (len(g), 3))
    v["normal"] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    v["uv"] = rng.uniform(0, 1, (len(g), 2))
    v["tangent"] = rng.uniform(-1, 1, (len(g), 3))
    i, j = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    a = (i * (side + 1) + j).reshape(-1)
    f = np.concatenate([np.stack([a, a + side + 1, a + 1], 1), np.stack([a + 1, a + side + 1, a + side + 2], 1)])
    return v, f[:n].astype(np.uint32)


def _builder(sizes, seed):
    rng = np.random.default_rng(seed)
    b = ag.SceneBuilder()
    b.add_point_light((0.0, 0.0, 6.0), (30.0, 28.0, 26.0))
    m = b.add_lambertian("m", (0.6, 0.5, 0.4))
    per = int(np.ceil(np.sqrt(len(sizes))))
    for k, n in enumerate(sizes):
        v, f = _patch(rng, n) if n else (np.zeros(3, A.VERTEX_DTYPE), np.zeros((0, 3), np.uint32))
        b.add_mesh(f"p{k}", v, f)
        t = np.eye(3, 4, dtype=np.float32)
        t[:, :3] *= np.float32(2.0 / per)
        t[:, 3] = (-1 + 2.0 * (k % per) / per, -1 + 2.0 * (k // per) / per, 0)
        b.add_instance(f"p{k}", m, t)
    return b


@pytest.mark.parametrize("sizes", [[4095], [4096], [4097], [4000, 0, 96], [1, 2, 4093, 3, 0], [6000, 10, 6000, 20],
                                   [10, 6000, 20, 6000, 0], [300] * 40, [255, 256, 257, 5000]])
def test_packed_meshes_render_like_the_oracle(ctx, sizes):
    b = _builder(sizes, len(sizes))
    state, depth = b.state(spp=2, max_path_depth=3, channels=("albedo", "normal", "position", "uv", "depth"))
    cam = ag.perspective_camera((0, 0, 3.0), (0, 0, 0), (0, 1, 0), 45.0, 40, 40)
    shot = ag.make_shot(cam, state, 40, 40, 2, depth_channel=depth)
    desc = b.desc()
    film = ctx.create_film(40, 40)
    ctx.render(ctx.create_scene(desc), shot, film)
    want, _, _ = oracle_py.OracleScene(desc).render(shot)
    for k in range(6):
        assert np.all(np.abs(film.read(k) - want[k]) <= 1e-4 * np.abs(want[k]) + 1e-6), k
    assert np.ptp(film.read(4)[..., 0]) > 0.1


@pytest.mark.parametrize("n", [100, 6000])
def test_index_out_of_range_is_refused(ctx, n):
    b = _builder([n, n], 1)
    b.meshes[1][1][3 * (n // 2) + 1] = len(b.meshes[1][0])
    with pytest.raises(A.AsunaError) as e:
        ctx.create_scene(b.desc())
    assert e.value.code == A.ERR_INVALID and "mesh 1: index" in str(e.value)
