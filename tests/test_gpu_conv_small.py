"""Convolutions of small images on the GPU: the tcgen05 kernel where a layer has
about as many units as the device has SMs (one-tile units, deep copy rings),
and the weight gradient's pipeline at few steps and part blocks; both against
float64."""
import ctypes as C

import numpy as np
import pytest

from asuna_gb300 import _abi as A
from oracle import unet_ref as U

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def bf16(a):
    return torch.from_numpy(np.asarray(a, np.float32)).cuda().to(torch.bfloat16).contiguous()


def run(name, *args):
    A.check(getattr(A.lib(), name)(None, *args))  # default stream: ordered with torch's own work
    torch.cuda.synchronize()


def p(t):
    return C.c_void_p(t.data_ptr())


# 1 unit with a ring that wraps (14 groups); 152 and 153 one-tile units; units
# of several tiles again (160 x 4 tiles); two channel slices of one tile
@pytest.mark.parametrize("shape", [(1, 16, 8, 224, 32), (1, 304, 64, 32, 16), (1, 17 * 16, 72, 16, 32),
                                   (5, 128, 128, 16, 16), (1, 5, 3, 48, 256)])
def test_tcgen05_units_about_the_sm_count(shape):
    n, h, w, cin, cout = shape
    rng = np.random.default_rng(h + w + cin)
    x = U.round_bf16(rng.normal(size=(n, h, w, cin)))
    wt = U.round_bf16(rng.normal(0, 0.2, (cout, 9, cin)))
    b = rng.normal(0, 0.1, cout).astype(np.float32)
    dx, dwt, db = bf16(x), bf16(wt), torch.from_numpy(b).cuda()
    wtc = torch.empty(cout * 9 * cin, dtype=torch.bfloat16, device="cuda")
    run("asuna_nn_weights_tc", p(dwt), p(wtc), cout, cin)
    out = torch.full((n, h, w, cout), float("nan"), dtype=torch.float32, device="cuda")
    run("asuna_nn_conv3x3_tc", p(dx), n, h, w, cin, p(wtc), p(db), cout, 0, None, p(out), 1)
    expired = C.c_int(-1)
    A.check(A.lib().asuna_nn_tc_status(C.byref(expired)))
    assert expired.value == 0
    ref = U.conv3x3(x, wt, b.astype(np.float64))
    # products of bf16 are exact in fp32; at most 9 x 224 + 1 additions of
    # relative error 2^-24 each, in the mean far fewer
    assert np.abs(out.cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()


# pixels: one step, the pipeline's depth and one more, part steps, part blocks
@pytest.mark.parametrize("shape", [(1, 1, 1, 16, 8), (1, 3, 32, 16, 16), (1, 4, 32, 80, 72), (1, 5, 32, 16, 64),
                                   (2, 13, 21, 48, 128), (1, 257, 1, 16, 32)])
def test_weight_gradient_pipeline(shape):
    n, h, w, cin, cout = shape
    rng = np.random.default_rng(h * w + cin)
    x = U.round_bf16(rng.normal(size=(n, h, w, cin)))
    dz = U.round_bf16(rng.normal(size=(n, h, w, cout)))
    ddz, dx = bf16(dz), bf16(x)
    dw = torch.zeros((cout, 9, cin), dtype=torch.float32, device="cuda")
    run("asuna_nn_conv3x3_wgrad", p(ddz), p(dx), n, h, w, cin, cout, p(dw))
    ref = U.conv3x3_dw(dz, x)
    assert np.abs(dw.cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()
