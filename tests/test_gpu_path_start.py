"""Rays started at their own triangle's leaf (the 2-wide ordered traversal)
against the skip-pointer walk: the occluder counts of AO do not depend on the
order in which leaves are visited, so both are equal exactly, for any triangle
a texel names, in either inner tree, alone and in a batch.  Thickness takes the
closest hit, where a hit in the face of its leaf's box may be met or not by that
order: equal but for single texels."""
import numpy as np
import pytest

from fornos_b200 import api
from fornos_b200 import workloads as W

pytestmark = pytest.mark.gpu

SPP, LO, HI = 33, 0.001, 0.4


def flat(quads, seed):
    rng = np.random.default_rng(seed)
    return W.grid_plane(quads, heights=0.1 * rng.uniform(0, 1, (quads + 1) ** 2))


# one leaf (no inner tree), one record, remainders, trees of many levels
@pytest.mark.parametrize("quads,max_tris", [(1, 8), (1, 1), (2, 8), (3, 1), (17, 3), (64, 8), (96, 1)])
@pytest.mark.parametrize("tree", [api.TREE_SAH, api.TREE_REFERENCE])
def test_path_start_equals_skip_walk(quads, max_tris, tree):
    ctx = api.Context(0)
    mesh = api.Mesh(flat(quads, quads))
    mesh.compute_vertex_normals()
    scene = api.Scene.build(ctx, mesh, max_tris)
    nt, n = 2 * quads * quads, 777
    rng = np.random.default_rng(5)
    # every seventh texel misses; the others start on a triangle of their own, some far outside it
    tidx = (3 * rng.integers(0, nt, n)).astype(np.uint32)
    tidx[:3] = 0, 3 * (nt - 1), 3 * (nt // 2)
    tidx[6::7] = api.MISS
    coords = np.zeros((n, 4), np.float32)
    coords[:, 1:] = rng.dirichlet((1, 1, 1), n)
    coords[1::5, 1:] = (3.0, -1.0, -1.0)
    scene.set_tree(tree)
    cb, tb = ctx.upload(coords), ctx.upload(tidx)
    table = ctx.upload(api.samples_cosine(SPP, 16, 3))
    got = []
    for traverse in (api.TRAVERSE_ORDERED, api.TRAVERSE_ORDERED | api.EXACT_BOX_TESTS, api.TRAVERSE_SKIP):
        out, hits = ctx.buffer(4 * n), ctx.buffer(4 * n)
        api.hemisphere(ctx, scene, cb, tb, api.AO, SPP, LO, HI, table, out, None, hits, None, 0, n, 16, traverse)
        got.append((out.download(np.uint32, n), hits.download(np.uint32, n)))
    jobs = [dict(scene=scene, coords=cb, tidx=tb, texel_count=n, spp=SPP, perms=16, min_distance=LO, max_distance=HI,
                 samples=table, out0=ctx.buffer(4 * n), hits0=ctx.buffer(4 * n)) for _ in range(2)]
    batch = api.Batch(ctx, jobs, api.AO)
    batch.run(api.TRAVERSE_ORDERED)
    got += [(j["out0"].download(np.uint32, n), j["hits0"].download(np.uint32, n)) for j in jobs]
    ctx.check()
    assert got[2][1].max() > 0 or nt <= 8
    for out, hits in got:
        assert np.array_equal(out, got[2][0]) and np.array_equal(hits, got[2][1])


@pytest.mark.parametrize("top", [1, 64, 608, 609, 640, 641, 768, 1024])
def test_staged_records_of_every_size(top):
    """Staged top records take the trace kernel's shared memory past the default
    limit within their allowed range; every size runs and gives the same counts."""
    ctx = api.Context(0)
    mesh = api.Mesh(flat(64, 3))
    mesh.compute_vertex_normals()
    scene = api.Scene.build(ctx, mesh, 1)
    n, nt = 500, 2 * 64 * 64
    rng = np.random.default_rng(6)
    coords = np.zeros((n, 4), np.float32)
    coords[:, 1:] = rng.dirichlet((1, 1, 1), n)
    cb, tb = ctx.upload(coords), ctx.upload((3 * rng.integers(0, nt, n)).astype(np.uint32))
    table = ctx.upload(api.samples_cosine(SPP, 16, 3))
    got = []
    for knobs, traverse in ((dict(top_records=top), api.TRAVERSE_ORDERED), (dict(top_records=0), api.TRAVERSE_SKIP)):
        ctx.set_tuning(**knobs)
        hits = ctx.buffer(4 * n)
        api.hemisphere(ctx, scene, cb, tb, api.AO, SPP, LO, HI, table, ctx.buffer(4 * n), None, hits, None, 0, n, 16,
                       traverse)
        got.append(hits.download(np.uint32, n))
    ctx.check()
    assert got[0].max() > 0 and np.array_equal(*got)


@pytest.mark.parametrize("shape", ["heights", "sphere"])
@pytest.mark.parametrize("tree", [api.TREE_SAH, api.TREE_REFERENCE])
def test_closest_hits_from_the_own_leaf(shape, tree):
    ctx = api.Context(0)
    mesh = api.Mesh(flat(64, 2) if shape == "heights" else W.sphere_pair(seed=2, hi_seg=(96, 48))[1])
    mesh.compute_vertex_normals()
    scene = api.Scene.build(ctx, mesh)
    scene.set_tree(tree)
    nt, n, hi = scene.info()["corner_count"] // 3, 3000, 3.0
    rng = np.random.default_rng(7)
    coords = np.zeros((n, 4), np.float32)
    coords[:, 1:] = rng.dirichlet((1, 1, 1), n)
    cb, tb = ctx.upload(coords), ctx.upload((3 * rng.integers(0, nt, n)).astype(np.uint32))
    table = ctx.upload(api.samples_cosine(SPP, 16, 3))
    got = []
    for traverse in (api.TRAVERSE_ORDERED, api.TRAVERSE_SKIP):
        out, hits = ctx.buffer(4 * n), ctx.buffer(4 * n)
        api.hemisphere(ctx, scene, cb, tb, api.THICK, SPP, LO, hi, table, out, None, hits, None, 0, n, 16, traverse)
        got.append((out.download(np.float32, n), hits.download(np.uint32, n)))
    ctx.check()
    assert 0.2 < (got[1][1] > 0).mean()
    # a hit met by one order alone changes its texel's mean of SPP distances by at most hi / SPP
    differ = got[0][0] != got[1][0]
    assert differ.mean() <= 1e-3 and np.all(np.abs(got[0][0] - got[1][0]) <= 2 * hi / SPP)
    assert np.array_equal(got[0][1][~differ], got[1][1][~differ])


def boxes(seed):
    """Closed boxes of flat, axis-aligned faces: leaves at faces of ancestors whose boxes round inward."""
    rng = np.random.default_rng(seed)
    g = W.grid_plane(6)
    parts = []
    for lo in rng.uniform(-1, 1, (8, 3)):
        size = rng.uniform(0.1, 0.8, 3)
        for axis in range(3):
            for side in (0, 1):
                p = np.zeros((len(g.positions), 3))
                p[:, (axis + 1) % 3], p[:, (axis + 2) % 3], p[:, axis] = g.positions[:, 0], g.positions[:, 1], side
                parts.append((lo + p * size)[g.triangles])
    n = 3 * sum(map(len, parts))
    return W.MeshArrays(np.concatenate(parts).reshape(-1, 3), np.zeros((1, 2)), [[0, 0, 1]],
                        np.stack([np.arange(n), np.zeros(n), np.zeros(n)], -1), np.arange(n).reshape(-1, 3))


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("kind", [api.AO, api.THICK])
def test_divided_box_tests_over_the_references_tree_equal_the_walk(seed, kind):
    """They reject exactly what the skip walk rejects, on meshes whose filtered
    traversal finds hits that the walk does not reach: hit counts are equal."""
    ctx = api.Context(0)
    mesh = api.Mesh(boxes(seed))
    mesh.compute_vertex_normals()
    scene = api.Scene.build(ctx, mesh)
    scene.set_tree(api.TREE_REFERENCE)
    nt, n = scene.info()["corner_count"] // 3, 3000
    rng = np.random.default_rng(seed)
    coords = np.zeros((n, 4), np.float32)
    coords[:, 1:] = rng.dirichlet((1, 1, 1), n)
    coords[1::3, 1:] = (0.5, 0.5, 0.0)
    cb, tb = ctx.upload(coords), ctx.upload((3 * rng.integers(0, nt, n)).astype(np.uint32))
    table = ctx.upload(api.samples_cosine(SPP, 16, 3))
    got = {}
    for name, traverse in (("walk", api.TRAVERSE_SKIP), ("divided", api.TRAVERSE_ORDERED | api.EXACT_BOX_TESTS),
                           ("filtered", api.TRAVERSE_ORDERED)):
        hits = ctx.buffer(4 * n)
        api.hemisphere(ctx, scene, cb, tb, kind, SPP, 0.0, 1.5, table, ctx.buffer(4 * n), None, hits, None, 0, n, 16,
                       traverse)
        got[name] = hits.download(np.uint32, n)
    job = dict(scene=scene, coords=cb, tidx=tb, texel_count=n, spp=SPP, perms=16, min_distance=0.0, max_distance=1.5,
               samples=table, out0=ctx.buffer(4 * n), hits0=ctx.buffer(4 * n))
    api.Batch(ctx, [job], kind).run(api.TRAVERSE_ORDERED | api.EXACT_BOX_TESTS)
    got["batch"] = job["hits0"].download(np.uint32, n)
    ctx.check()
    assert not np.array_equal(got["filtered"], got["walk"])  # the mesh shows the difference
    assert np.array_equal(got["divided"], got["walk"]) and np.array_equal(got["batch"], got["walk"])
