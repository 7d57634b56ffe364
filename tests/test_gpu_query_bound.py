"""A ray query that passes the traversal's loop bound (65,536 leaves and
instances of one ray) reports it, as a render does."""
import numpy as np
import pytest

from asuna_gb300 import _abi as A
from asuna_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("any_hit", [False, True])
def test_runaway_query_is_reported(ctx, any_hit):
    b, _ = scenes.stacked_instances_scene(70000)
    scene = ctx.create_scene(b.desc())
    o, d = np.array([[5.0, 0.0, 3.0], [0.9, 0.9, 3.0]], np.float32), np.array([[0, 0, -1.0]] * 2, np.float32)
    hits, inst = scene.trace(o[:1], d[:1], any_hit=any_hit)  # past every box
    assert hits[0, 0] == -1.0 and inst[0] == 0xFFFFFFFF
    with pytest.raises(A.AsunaError) as e:
        scene.trace(o, d, any_hit=any_hit)  # the second one misses each triangle, inside its box
    assert e.value.code == A.ERR_TRAVERSAL
    b, _ = scenes.stacked_instances_scene(300)
    hits, inst = ctx.create_scene(b.desc()).trace(o, d, any_hit=any_hit)
    assert np.all(inst == 0xFFFFFFFF)
