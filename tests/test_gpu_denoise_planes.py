"""The denoiser's layers with their neighbours fused (pooling, upsampling, the
output image) over ragged sizes, batches and depths: against the float64
network with bf16 storage, and bit for bit between handles and batch sizes."""
import numpy as np
import pytest

import asuna_gb300 as ag
from asuna_gb300 import denoise as dn
from oracle import unet_ref as U

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def dctx():
    return ag.Context(0)


@pytest.mark.parametrize("ch", [(16, 32), (32, 48, 64), dn.DEFAULT_CHANNELS])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 17, 9), (2, 33, 70)])
def test_fused_layers(dctx, ch, shape):
    n, h, w = shape
    rng = np.random.default_rng(h * w + len(ch))
    rad = rng.gamma(1.2, 0.5, (n, h, w, 4)).astype(np.float32)
    alb = rng.uniform(0, 1, (n, h, w, 4)).astype(np.float32)
    nrm = rng.normal(size=(n, h, w, 4)).astype(np.float32)
    wsum = np.repeat(rng.uniform(1.0, 600.0, (n, h, w, 1)), 4, axis=3).astype(np.float32)
    p = U.he_init(ch, 6)
    p = (p + rng.normal(0, 0.02, p.size)).astype(np.float32)
    outs = {}
    for training in (False, True):
        for tm in (False, True):
            d = dn.Denoiser(dctx, ch, seed=3, max_pixels=n * 48 * 96, training=training, tensor_memory=tm)
            d.set_params(p)
            g = [torch.from_numpy(a).cuda() for a in (rad, alb, nrm, wsum)]
            torch.cuda.synchronize()
            out = d.forward(*g)
            dctx.sync()
            outs[training, tm] = out.cpu().numpy()
            if tm and not training:
                for i in range(n):
                    one = d.forward(*[t[i:i + 1].contiguous() for t in g])
                    dctx.sync()
                    assert np.array_equal(one.cpu().numpy()[0], outs[False, True][i])
    ro = U.UNetRef(ch, p, bf16=True).output(rad.astype(np.float64), alb, nrm, wsum, None)
    for tm in (False, True):
        # what a training handle keeps besides does not change the output
        assert np.array_equal(outs[False, tm], outs[True, tm])
        got = outs[False, tm][..., :3]
        # accumulation order only: a sum on the other side of a bf16 step (2^-8)
        # in a few of the activations
        assert np.median(np.abs(got - ro) / (np.abs(ro) + 1e-3)) < 5e-3
        assert np.abs(got - ro).max() <= 0.05 * np.abs(ro).max()
        assert np.all(outs[False, tm][..., 3] == 1.0)


@pytest.mark.parametrize("ch", [(16, 16), (32, 256), (48, 64, 192)])
def test_gradients_with_sliced_weights(dctx, ch):
    """Loss and gradients on tcgen05 against mma.sync, where layers have one
    and several weight slices in either direction."""
    n, h, w = 2, 19, 26
    rng = np.random.default_rng(sum(ch))
    rad = rng.gamma(1.2, 0.5, (n, h, w, 4)).astype(np.float32)
    tgt = (rad * rng.uniform(0.5, 1.5, rad.shape)).astype(np.float32)
    p = U.he_init(ch, 6)
    p = (p + rng.normal(0, 0.02, p.size)).astype(np.float32)
    res = []
    for tm in (False, True):
        d = dn.Denoiser(dctx, ch, seed=3, max_pixels=n * 32 * 32, training=True, tensor_memory=tm)
        d.set_params(p)
        grad, gtgt = torch.from_numpy(rad).cuda(), torch.from_numpy(tgt).cuda()
        torch.cuda.synchronize()
        res.append((d.loss_grad(grad, None, None, None, gtgt), d.get_grads().astype(np.float64)))
    (l0, g0), (l1, g1) = res
    # bounds as for the default network: accumulation order before bf16 rounding
    assert abs(l1 - l0) <= 1e-3 * l0
    assert np.linalg.norm(g1 - g0) < 0.03 * np.linalg.norm(g0)
