"""The tcgen05 convolution's bounded waits cover its own copies and MMAs only: in
a chain of layers, every role waits for the layer before (which may take any
time) ahead of its first bounded wait, and the MMA warp looks at the error of
the layer before only then.  Whether a wait's bound is passed depends on the
chip's load, so the order is read from the source; on the GPU, a batch whose
layers run far longer than an image's own gives the images one by one, with no
wait expired."""
import ctypes as C
import os
import re

import numpy as np
import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "asuna_gb300", "csrc", "conv_tc.cu")


def _roles():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    body = text[text.index("k_conv_tc("):]
    body = body[:body.index("\n}\n")]
    producer = body.index("if (warp == kProducerWarp)")
    mma = body.index("} else if (warp == kMmaWarp) {")
    epilogue = body.index("\n  } else {", mma)
    return {"producer": body[producer:mma], "mma": body[mma:epilogue], "epilogue": body[epilogue:]}


@pytest.mark.parametrize("role", ["producer", "mma", "epilogue"])
def test_previous_layer_is_waited_for_first(role):
    body = re.sub(r"auto waitAll = .*?};", "", _roles()[role], flags=re.S)
    waits = [m.start() for m in re.finditer(r"mbarWaitOr\(|waitAll\(", body)]
    assert waits and "waitForPrevious()" in body
    assert body.index("waitForPrevious()") < min(waits)


def test_error_of_the_previous_layer_is_read_after_it():
    body = _roles()["mma"]
    assert body.index("waitForPrevious()") < body.index("g_tcError") < body.index("mma(acc")


@pytest.mark.gpu
def test_long_layers_equal_single_images():
    torch = pytest.importorskip("torch")
    import asuna_gb300 as ag
    from asuna_gb300 import _abi as A
    from asuna_gb300 import denoise as dn

    n, h, w = 12, 544, 960
    ctx = ag.Context(0)
    rng = np.random.default_rng(5)
    rad = torch.from_numpy(rng.gamma(1.2, 0.5, (n, h, w, 4)).astype(np.float32)).cuda()
    alb = torch.from_numpy(rng.uniform(0, 1, (n, h, w, 4)).astype(np.float32)).cuda()
    d = dn.Denoiser(ctx, seed=3, max_pixels=n * h * w)
    torch.cuda.synchronize()
    batch = d.forward(rad, alb)
    ctx.sync()
    for i in (0, n - 1):
        one = d.forward(rad[i:i + 1].contiguous(), alb[i:i + 1].contiguous())
        ctx.sync()
        assert torch.equal(one[0], batch[i])
    expired = C.c_int(-1)
    A.check(A.lib().asuna_nn_tc_status(C.byref(expired)))
    assert expired.value == 0
    ctx.close()
