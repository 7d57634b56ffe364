"""Speculating lanes and the traversal stack: a speculative node step keeps an
older leaf group on the stack as well, and must leave room for the rest of the
tree.  Whatever number of entries the ordered traversal gets by with is enough
for the speculating one, in ordinary trees and in a mesh nested so deep that
its wide tree is a chain of some thirty levels; the full stack fits both."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import _abi as A
from asuna_gb300 import scenes

pytestmark = pytest.mark.gpu



def _nested(levels=33, ratio=2.5, per=32, inner=1e-4):
    """Clusters of slivers, each `ratio` times the size of the one inside: every
    wide node is filled by a cluster's parts, and the rest hangs one level down.
    The camera sits at the inner end, with the clusters in one half of its view
    and a cloud of specks in the other, so that half of a warp's lanes walk
    through inner nodes while the others have leaves in hand."""
    rng = np.random.default_rng(1)
    tris = []
    for k in range(levels):
        s = inner * ratio ** k
        lo, hi = np.array([1 / ratio, 0, 0]) * s, np.array([1.0, 1, 1]) * s
        a, b = rng.uniform(0, 0.05, (per, 3)), rng.uniform(0.95, 1, (per, 3))
        flip = rng.random((per, 3)) < 0.5
        a, b = lo + np.where(flip, b, a) * (hi - lo), lo + np.where(flip, a, b) * (hi - lo)
        tris.append(np.stack([a, b, b + rng.normal(size=(per, 3)) * 1e-4 * s], 1))
    specks = rng.uniform(-1, 1, (100000, 1, 3)) * [1, 4, 4] - [4, 0, 0] + rng.normal(size=(100000, 3, 3)) * 1e-3
    b = ag.SceneBuilder()
    m = b.add_lambertian("m", (0.5, 0.5, 0.5))
    for name, t in (("nested", np.concatenate(tris)), ("specks", specks)):
        v = np.zeros(3 * len(t), A.VERTEX_DTYPE)
        v["pos"] = t.reshape(-1, 3).astype(np.float32)
        v["normal"] = (0, 0, 1)
        b.add_mesh(name, v, np.arange(len(v), dtype=np.uint32))
        b.add_instance(name, m)
    b.add_point_light((-1.0, -1.0, 2.0), (10.0, 10.0, 10.0))
    state, _ = b.state(spp=1, max_path_depth=2, channels=())
    w, h = 32, 4096  # a row of pixels is a warp
    eye = np.full(3, -inner)
    cam = ag.opencv_camera(eye, eye + [0, 1, 1], (0, -1, 1), (w / 3.4, h / 1.2, w / 2, h / 2))
    return b, ag.make_shot(cam, state, w, h, 1)


def _mixed():
    return scenes.mixed_scene(512, 256, frames=1, max_depth=4, n_spheres=16, level=5, seed=4, env_size=(32, 16))


# (more paths than the path kernel takes: the passes speculate)
@pytest.mark.parametrize("make", [_mixed, _nested])
def test_speculation_needs_no_more_entries(ctx, make):
    b, shot = make()
    scene, film = ctx.create_scene(b.desc()), ctx.create_film(shot.width, shot.height)

    def fits(entries, speculate):
        ctx.set_traversal(speculate_extend=speculate, speculate_shadow=speculate)
        ctx.set_traversal_stack(entries)
        try:
            film.clear()
            ctx.render(scene, shot, film, stats=True)
            return True
        except A.AsunaError as e:
            assert e.code == A.ERR_TRAVERSAL
            return False
        finally:
            ctx.set_traversal()
            ctx.set_traversal_stack(0)

    assert fits(0, 0)
    want = film.read(0)
    lo, hi = 0, 64  # cut short with lo entries, not with hi
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid, 0) else (mid, hi)
    assert 3 <= hi < 64
    for entries in [*range(hi, min(hi + 8, 64)), 0]:
        assert fits(entries, 1), (entries, hi)
        assert np.array_equal(film.read(0), want)
    if make is _nested:
        assert hi > 15
