"""The per-texel folds of the dynamic schedule against the static schedule's,
which folds in its own kernel: the same walk, so the same bits, for sample counts
round the folds' step of 8 and their switch at 32, texel counts that leave
warps part full, misses, and texel lists."""
import numpy as np
import pytest

from fornos_b200 import api
from fornos_b200 import workloads as W

pytestmark = pytest.mark.gpu

KINDS = {"ao": api.AO, "bn": api.BN, "thickness": api.THICK, "ao_bn": api.AO_BN}


@pytest.fixture(scope="module")
def scene():
    ctx = api.Context(0)
    mesh = api.Mesh(W.plane_pair(seed=6, hi_quads=24, bumps=10)[1])
    mesh.compute_vertex_normals()
    return ctx, api.Scene.build(ctx, mesh), 2 * 24 * 24


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("spp,n", [(1, 33), (7, 300), (31, 257), (32, 1), (33, 95), (40, 256), (64, 129), (100, 31)])
def test_fold_equals_static_schedule(scene, kind, spp, n):
    ctx, sc, nt = scene
    rng = np.random.default_rng(spp)
    tidx = (3 * rng.integers(0, nt, n)).astype(np.uint32)
    tidx[3::5] = api.MISS
    coords = np.zeros((n, 4), np.float32)
    coords[:, 1:] = rng.dirichlet((1, 1, 1), n)
    cb, tb = ctx.upload(coords), ctx.upload(tidx)
    table = ctx.upload(api.samples_cosine(spp, 16, 3))

    def run(schedule, ids=None):
        k = KINDS[kind]
        out = [ctx.buffer(12 * n) for _ in range(2)] + [ctx.buffer(4 * n) for _ in range(2)]
        args = (ctx, sc, cb, tb)
        rest = (k, spp, 0.001, 0.3, table)
        if ids is None:
            api.hemisphere(*args, *rest, *out, 0, n, 16, api.TRAVERSE_SKIP | schedule)
        else:
            api.hemisphere_texels(*args, n, *rest, ctx.upload(ids), *out, 0, n, 16, api.TRAVERSE_SKIP | schedule)
        return [b.download(np.uint32, b.nbytes // 4) for b in out]

    want = run(api.SCHEDULE_STATIC)
    for got in (run(api.SCHEDULE_DYNAMIC), run(api.SCHEDULE_DYNAMIC, rng.permutation(n).astype(np.uint32))):
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    ctx.check()
