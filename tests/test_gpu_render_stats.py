"""Timing fields of the render statistics: the traversal fields hold the
traversal kernels alone, and a wave that the path kernel takes is timed as
that kernel's."""
import pytest

from asuna_gb300 import scenes

pytestmark = pytest.mark.gpu


def _render(ctx, size):
    b, shot = scenes.mixed_scene(*size, frames=1, max_depth=5, n_spheres=6, level=3, seed=3, env_size=(32, 16))
    scene, film = ctx.create_scene(b.desc()), ctx.create_film(*size)
    ctx.render(scene, shot, film)
    return ctx.render(scene, shot, film, stats=True)


@pytest.mark.parametrize("graphs", [True, False])
def test_path_kernel_is_a_kind_of_its_own(ctx, graphs):
    ctx.set_graphs(graphs)
    try:
        small, large = _render(ctx, (128, 96)), _render(ctx, (512, 256))
    finally:
        ctx.set_graphs(True)
    assert small["extend_launches"] == small["connect_launches"] == 0
    assert small["ms_extend"] == small["ms_connect"] == small["ms_shade"] == small["ms_sort"] == 0.0
    assert small["path_launches"] == 1 and 0.0 < small["ms_path"] <= small["ms_total"]
    assert small["extend_rays"] > small["paths"]
    # passes 1 to 5 are issued; from the second on the path kernel looks first
    assert large["extend_launches"] == large["connect_launches"] == 5 and large["path_launches"] == 4
    parts = [large[k] for k in ("ms_extend", "ms_shade", "ms_connect", "ms_path")]
    assert min(parts) > 0.0 and sum(parts) <= large["ms_total"]
