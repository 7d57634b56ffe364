"""The path kernel against pure wavefront passes (the instrumented traversal
runs those): films are bit-identical around the number of rays at which it
takes over, from the first pass or in a later one, through the graph's loop,
without a graph, with the queue sort, and in records; with pass-through
surfaces (which need passes beyond the depth limit) and without."""
import numpy as np
import pytest

from asuna_gb300 import scenes

pytestmark = pytest.mark.gpu

SIZES = {"plugins": [(1, 1), (50, 40), (192, 128), (193, 128), (260, 200)],
         "mixed": [(1, 3), (64, 48), (384, 256), (385, 256), (500, 400)]}


def _films(film):
    return np.stack([film.read(k) for k in (0, 1, 2, 3, 8)])


@pytest.mark.parametrize("kind,size,opacity", [(k, s, o) for k in SIZES for s in SIZES[k]
                                               for o in ((False, True) if k == "plugins" else (False,))])
def test_films_equal_wavefront_films(ctx, kind, size, opacity):
    w, h = size
    if kind == "plugins":
        b, shot = scenes.plugin_scene(w, h, frames=1, max_depth=6, channels=("albedo", "normal", "depth"),
                                      textured=True, opacity=opacity)
    else:
        b, shot = scenes.mixed_scene(w, h, frames=1, max_depth=7, n_spheres=6, level=3, seed=3, env_size=(32, 16))
    scene, film = ctx.create_scene(b.desc()), ctx.create_film(w, h)
    ctx.set_counters(True)
    try:
        ctx.render(scene, shot, film)
        want = _films(film)
        rays = ctx.render(scene, shot, film, stats=True)
    finally:
        ctx.set_counters(False)
    assert np.isfinite(want).all() and want[0, ..., :3].max() > 0
    for graphs, sort in ((True, 0), (False, 0), (True, 3), (False, 3)):
        ctx.set_graphs(graphs)
        ctx.set_ray_sort(sort)
        try:
            for _ in range(2):  # recorded, then replayed
                film.clear()
                ctx.render(scene, shot, film)
                assert np.array_equal(_films(film), want), (graphs, sort)
            st = ctx.render(scene, shot, film, stats=True)
            assert (st["extend_rays"], st["shadow_rays"], st["paths"]) == \
                (rays["extend_rays"], rays["shadow_rays"], rays["paths"])
        finally:
            ctx.set_graphs(True)
            ctx.set_ray_sort(0)
    film.clear()
    rec = ctx.render_paths(scene, shot, film)
    assert np.array_equal(_films(film), want)
    assert rec["depth"].max() > 1 or w * h < 10


def test_batch_of_waves_of_both_kinds(ctx):
    """A path budget that cuts a batch into waves above and below the path
    kernel's size gives the films of single renders."""
    b, _ = scenes.mixed_scene(8, 8, frames=1, n_spheres=6, level=3, seed=3, env_size=(32, 16))
    scene = ctx.create_scene(b.desc())
    sizes = [(400, 300, 2), (40, 30, 3), (300, 200, 1), (7, 5, 2)]
    shots = [scenes.mixed_shot(b, w, h, f, max_depth=6, seed=k) for k, (w, h, f) in enumerate(sizes)]
    single = []
    for s in shots:
        film = ctx.create_film(s.width, s.height)
        ctx.render(scene, s, film)
        single.append(film.read(0))
    ctx.set_path_budget(1)  # one frame of the largest shot at a time
    try:
        films = [ctx.create_film(s.width, s.height) for s in shots]
        ctx.render_batch(scene, shots, films)
        for f, want in zip(films, single):
            assert np.array_equal(f.read(0), want)
    finally:
        ctx.set_path_budget(0)
