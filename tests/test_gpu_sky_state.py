"""The sky's direction-independent state, evaluated once per scene: films under
suns above, at and below the horizon, with every optional part on and off,
equal the oracle's (which evaluates it per direction with the same operations)
within the bound of the other film comparisons."""
import numpy as np
import pytest

from asuna_gb300 import scenes
from oracle import oracle_py

pytestmark = pytest.mark.gpu

CASES = [dict(), dict(sun_direction=(0.1, 0.001, 0.9)), dict(sun_direction=(0.5, -0.2, 0.5)),
         dict(sun_direction=(0.0, -1.0, 0.1)), dict(multiplier=0.0), dict(multiplier=-1.0),
         dict(sun_disk_intensity=0.0), dict(sun_disk_scale=0.0), dict(physically_scaled_sun=0, haze=7.0),
         dict(horizon_blur=0.0, horizon_height=0.4), dict(y_is_up=0, saturation=0.2, redblueshift=-0.3),
         dict(rgb_unit_conversion=(-1.0, -1.0, -1.0), haze=-5.0), dict(saturation=1.7, night_color=(0.2, 0.1, 0.3))]


@pytest.mark.parametrize("fields", CASES)
@pytest.mark.parametrize("dusk", [False, True])
def test_sky_film_matches_oracle(ctx, fields, dusk):
    b, shot = scenes.sky_scene(24, 18, frames=2, max_depth=4, dusk=dusk)
    b.set_sun_and_sky(**fields)
    desc = b.desc()
    film = ctx.create_film(24, 18)
    ctx.render(ctx.create_scene(desc), shot, film)
    want, _, _ = oracle_py.OracleScene(desc).render(shot)
    got = film.read(0)
    assert np.array_equal(np.isfinite(got), np.isfinite(want[0]))
    ok = np.isfinite(want[0])
    assert np.all(np.abs(got - want[0])[ok] <= (1e-4 * np.abs(want[0]) + 1e-6)[ok])
