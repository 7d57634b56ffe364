"""Environment importance tables made on the device: films lit by maps around
the size from which they are, with rows and columns off the warp size, single
rows and columns, black rows and zero maps, equal the oracle's (which builds
its own tables on the host) within the bound of the other film comparisons:
one table entry that differs sends samples elsewhere."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import scenes
from oracle import oracle_py

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,kind", [(64, 63, "noise"), (64, 64, "noise"), (65, 64, "noise"), (131, 67, "noise"),
                                      (512, 256, "noise"), (5000, 1, "noise"), (1, 5000, "noise"), (97, 101, "rows"),
                                      (128, 64, "zero"), (31, 200, "noise"), (300, 40, "flat")])
def test_film_under_a_map_matches_oracle(ctx, w, h, kind):
    rng = np.random.default_rng(w * 7919 + h)
    env = rng.lognormal(0.0, 1.5, (h, w, 4)).astype(np.float32)
    if kind == "rows":
        env[rng.random(h) < 0.5] = 0.0
    elif kind == "zero":
        env[:] = 0.0
    elif kind == "flat":
        env[:] = 0.5
    b = ag.SceneBuilder()
    b.set_envmap(env)
    m = b.add_lambertian("m", (0.7, 0.6, 0.5))
    v, f = scenes.icosphere(2)
    verts = np.zeros(len(v), ag._abi.VERTEX_DTYPE)
    verts["pos"], verts["normal"] = v, v
    b.add_mesh("s", verts, f.astype(np.uint32))
    b.add_instance("s", m)
    state, _ = b.state(spp=4, max_path_depth=3)
    cam = ag.perspective_camera((0, 0, 3.0), (0, 0, 0), (0, 1, 0), 60.0, 40, 32)
    shot = ag.make_shot(cam, state, 40, 32, 4)
    desc = b.desc()
    film = ctx.create_film(40, 32)
    ctx.render(ctx.create_scene(desc), shot, film)
    want, _, _ = oracle_py.OracleScene(desc).render(shot)
    assert np.all(np.abs(film.read(0) - want[0]) <= 1e-4 * np.abs(want[0]) + 1e-6)
