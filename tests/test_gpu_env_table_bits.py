"""Environment importance tables made on the device equal the host's
(asuna_envmap_tables) entry by entry and bit for bit, around the size from
which the device makes them and off the warp size, with black rows, a zero map,
equal texels, fireflies, negative and denormal texels."""
import platform

import numpy as np
import pytest

import asuna_gb300 as ag

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(platform.machine() != "aarch64", reason="the host compiler fuses the texel weight on Arm only")
@pytest.mark.parametrize("w,h,kind", [(64, 63, "noise"), (64, 64, "noise"), (65, 64, "noise"), (131, 67, "noise"),
                                      (512, 256, "noise"), (1024, 512, "noise"), (5000, 1, "noise"),
                                      (1, 5000, "noise"), (97, 101, "rows"), (128, 64, "zero"), (300, 40, "flat"),
                                      (200, 33, "fireflies"), (100, 50, "negative"), (100, 50, "denormal")])
def test_tables_equal_the_hosts(ctx, w, h, kind):
    rng = np.random.default_rng(w * 7919 + h)
    env = rng.lognormal(0.0, 1.5, (h, w, 4)).astype(np.float32)
    if kind == "rows":
        env[rng.random(h) < 0.5] = 0.0
    elif kind == "zero":
        env[:] = 0.0
    elif kind == "flat":
        env[:] = 0.5
    elif kind == "fireflies":
        env[rng.random((h, w)) < 0.01] *= 1e20
    elif kind == "negative":
        env[rng.random((h, w)) < 0.1] *= -1.0
    elif kind == "denormal":
        env *= 1e-42
    b = ag.SceneBuilder()
    b.set_envmap(env)
    b.add_lambertian("m", (0.7, 0.6, 0.5))
    marg, cond = ctx.create_scene(b.desc()).envmap_tables(w, h)
    want_marg, want_cond = ag.envmap_tables(env)
    for got, want in ((marg, want_marg), (cond, want_cond)):
        got, want = got.reshape(-1).view(np.uint32), np.ascontiguousarray(want).reshape(-1).view(np.uint32)
        assert got.shape == want.shape and np.array_equal(got, want)
