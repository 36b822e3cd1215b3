"""The tcgen05 engine's positions over a texel's spacing against the mma.sync
engine's, which divides: spacings inside and outside the range of the reciprocal
form, positions that are huge, infinite or equal.  Both engines round the features
and activations to bf16; the bar is that of the other engine comparisons (a value
at a rounding boundary may round either way)."""
import numpy as np
import pytest

from fornos_b200 import api
from fornos_b200.denoise_train import init_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [1e-3, 1.0, 1e-19, 1e-25, 1e19, 1e-38, 3e38])
def test_engines_agree_over_spacings(spacing):
    ctx = api.Context(0)
    w, h = 37, 19
    n = w * h
    rng = np.random.default_rng(4)
    image = np.zeros((3, n, 4), np.float32)
    image[0, :, :3] = rng.uniform(-1, 1, (n, 3))
    image[0, :, 3] = rng.uniform(0, 1, n) > 0.1
    with np.errstate(over="ignore"):
        image[1, :, :3] = (rng.normal(size=(n, 3)) * 2 * spacing).astype(np.float32)
    image[1, 5::50, 0] = np.inf
    image[1, 7::50, 1] = 3e38
    image[1, 9::50, 2] = image[1, 8::50, 2][:len(image[1, 9::50, 2])]
    image[1, :, 3] = rng.uniform(0, 1, n)
    image[2, :, :2] = rng.uniform(-1, 1, (n, 2))
    image[2, :, 2] = np.float32(spacing) * rng.uniform(0.5, 1.0, n).astype(np.float32)
    image[2, 11::60, 2] = 0.0
    tmap = api.TexelMap.from_host(ctx, w, h, np.zeros((n, 8)), np.zeros((n, 12)), np.arange(n))
    img, tidx = ctx.upload(image), ctx.upload(np.zeros(n, np.uint32))
    ao, bn = ctx.upload(rng.uniform(0, 1, n).astype(np.float32)), ctx.upload(rng.normal(size=(n, 3)).astype(np.float32))
    net = api.Denoiser(ctx, init_params(3))
    got = []
    for engine in (api.DN_ENGINE_MMA_SYNC, api.DN_ENGINE_TCGEN05):
        net.set_engine(engine)
        out_ao, out_bn = ctx.buffer(4 * n), ctx.buffer(12 * n)
        net.apply(tmap, img, tidx, ao, bn, out_ao, out_bn)
        got.append(np.concatenate([out_ao.download(np.float32, n), out_bn.download(np.float32, 3 * n)]))
    ctx.check()
    assert np.array_equal(np.isnan(got[0]), np.isnan(got[1]))
    d = np.abs(np.nan_to_num(got[0]) - np.nan_to_num(got[1]))
    assert np.quantile(d, 0.99) < 1e-5 and d.max() < 2e-3
