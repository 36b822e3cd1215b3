"""Mesh mapping over the inner tree against the skip-pointer walks, bit for
bit.  A direction eight times as long takes the walks (the tree route asks for
about unit length) and every operation on it is the same but for an exact power
of two, so both routes run on the same rays and distances differ by that
factor alone.  That the tree answered the unit directions is counted."""
import numpy as np
import pytest

from fornos_b200 import api
from fornos_b200 import workloads as W
from tests.cases import bits

pytestmark = pytest.mark.gpu


def soup(n, seed, size, thin=None, scale=1.0, shift=(0.0, 0.0, 0.0), slivers=False):
    """Triangles of all shapes: ordinary ones, thin ones (down to the angle
    `thin`), repeated corners, collinear corners, identical triangles, one as
    large as the scene; with `slivers` thinner than any bound allows."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    p = (c + size * rng.normal(size=(n, 3, 3))).astype(np.float32)
    if slivers:
        p[1::7, 2] = p[1::7, 1] + (p[1::7, 0] - p[1::7, 1]) * np.float32(1e-3) + np.float32(1e-6)
        p[3::7, 2] = 0.5 * (p[3::7, 0] + p[3::7, 1])
    else:
        v0, v1 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        up = np.cross(v0, v1)
        up /= np.linalg.norm(up, axis=1, keepdims=True)
        across = np.cross(up, v0)  # of v0's length, at a right angle to it in the triangle's plane
        sin = np.linalg.norm(np.cross(v0, v1), axis=1) / (np.linalg.norm(v0, axis=1) * np.linalg.norm(v1, axis=1))
        p[:, 2] = np.where((sin < 0.1)[:, None], p[:, 0] + across, p[:, 2])
        if thin:
            a = np.exp(rng.uniform(np.log(thin), 0, n))[:, None]
            p[1::7, 2] = (p[:, 0] + v0 * np.cos(a) + across * np.sin(a))[1::7]
        # collinear to the last bit: grid points with the third corner twice as far as the second
        q, g = (p[3::7, 0] * 64).round() / 64, (v0[3::7] * 256).round() / 256
        p[3::7] = np.stack([q, q + g, q + 2 * g], 1)
    p[2::7, 2] = p[2::7, 1]
    p[4::14] = p[4]
    p[-1] = [[-1, -1, 0], [1, -1, 0], [0, 1, 0]]
    p = p * np.float32(scale) + np.asarray(shift, np.float32)
    tri = np.arange(3 * n).reshape(-1, 3)
    return W.MeshArrays(p.reshape(-1, 3), np.zeros((1, 2)), np.tile([[0, 0, 1]], (3 * n, 1)),
                        np.stack([np.arange(3 * n), np.zeros(3 * n), np.arange(3 * n)], -1), tri)


MESHES = {
    "sphere": lambda: W.sphere_pair(seed=3, hi_seg=(256, 96))[1],     # thin triangles round the poles
    "heights": lambda: W.plane_pair(seed=4, hi_quads=64, bumps=20)[1],
    "flat": lambda: W.grid_plane(32),                                 # every hit lies in its leaf's box face
    "soup": lambda: soup(4000, 5, 0.02),
    "thin_soup": lambda: soup(4000, 9, 0.02, thin=4e-4),
    "coarse_soup": lambda: soup(300, 6, 0.4),
    "small_soup": lambda: soup(1000, 10, 0.05, scale=2.0 ** -9, shift=(0.5, -0.25, 0.125)),
    "large_soup": lambda: soup(1000, 11, 0.05, scale=64.0, shift=(100.0, -300.0, 50.0)),
    "two": lambda: W.grid_plane(1),                             # a single leaf has no tree
    "nine": lambda: soup(9, 7, 0.3),
    "slivers": lambda: soup(4000, 5, 0.02, slivers=True),       # no bound: the walks throughout
    "nine_slivers": lambda: soup(9, 7, 0.3, slivers=True),
}


def rays(mesh, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = mesh.positions.min(0), mesh.positions.max(0)
    o = rng.uniform(lo - 0.05, hi + 0.05, (n, 3))
    d = rng.normal(size=(n, 3))
    d[::3] = np.eye(3)[rng.integers(0, 3, len(d[::3]))] * rng.choice([-1, 1], (len(d[::3]), 1))  # along the axes
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    # on the mesh: at corners, on edges and inside triangles (axis-aligned rays there run in box faces)
    p = mesh.positions[mesh.vertices[mesh.triangles, 0]].astype(np.float64)
    w = rng.dirichlet((1, 1, 1), n)
    w[1::4] = (0.5, 0.5, 0.0)
    w[2::4] = (1.0, 0.0, 0.0)
    on = (p[rng.integers(0, len(p), n)] * w[:, :, None]).sum(1)
    o[::2] = on[::2] + rng.choice([0, 0.01, -0.01], (len(on[::2]), 1)) * d[::2]
    o[5] = 100.0  # far outside
    d[7, 0] = np.nan
    o[11, 1] = np.nan
    return o.astype(np.float32), d.astype(np.float32)


def texel_map(ctx, o, d):
    n = len(o)
    pix = np.zeros((n, 8), np.float32)
    pix[:, 0:3], pix[:, 4:7] = o, d
    return api.TexelMap.from_host(ctx, n, 1, pix, np.zeros((n, 12), np.float32), np.arange(n))


def mapped(ctx, scene, o, d, cull, max_d):
    n = len(o)
    tmap = texel_map(ctx, o, d)
    coords, tidx = ctx.buffer(16 * n), ctx.buffer(4 * n)
    api.meshmap(ctx, scene, tmap, cull, coords, tidx, max_dist=max_d)
    return coords.download(np.float32, (n, 4)), tidx.download(np.uint32, n)


@pytest.mark.parametrize("name", sorted(MESHES))
@pytest.mark.parametrize("cull", [True, False])
def test_tree_route_equals_walks(name, cull):
    ctx = api.Context(0)
    arrays = MESHES[name]()
    mesh = api.Mesh(arrays)
    mesh.compute_vertex_normals()
    scene = api.Scene.build(ctx, mesh)
    o, d = rays(arrays, 4099, 8)
    for max_d, tree in ((api.FLT_MAX, api.TREE_SAH), (0.25, api.TREE_REFERENCE)):
        scene.set_tree(tree)  # the mapping does not depend on the active tree
        c1, t1 = mapped(ctx, scene, o, d, cull, max_d)
        c8, t8 = mapped(ctx, scene, o, 8 * d, cull, max_d if max_d == api.FLT_MAX else max_d / 8)
        hit = t1 != api.MISS
        by_tree, _ = api.meshmap_routes(ctx, scene, texel_map(ctx, o, d), cull, max_d)
        walked, _ = api.meshmap_routes(ctx, scene, texel_map(ctx, o, 8 * d), cull, max_d)
        assert walked == 0
        assert by_tree == 0 if "slivers" in name or name == "two" else by_tree > 0.8 * len(o)
        assert np.array_equal(t1, t8)
        # as bits: a texel on a triangle seen from behind maps to -0
        assert np.array_equal(bits(c1[hit, 0]), bits(8 * c8[hit, 0]))
        assert np.array_equal(bits(c1[:, 1:]), bits(c8[:, 1:]))
        assert hit.sum() > 100 or name in ("two", "nine", "nine_slivers", "flat")
    ctx.check()


@pytest.mark.parametrize("cull", [True, False])
def test_leaves_in_another_order_than_their_corners(cull):
    """Among hits at one distance the walks keep the first they meet, which is
    the smallest corner only where the leaves' corners ascend: an uploaded tree
    whose leaves name them in descending order, on the edges between leaves."""
    quads, n = 16, 4000
    mesh = api.Mesh(W.grid_plane(quads))
    built = api.BVH.create_binary(mesh).flatten(mesh)
    nodes, pos4, nrm4 = (a.copy() for a in built)
    order, at = [], 0
    for i in np.flatnonzero(nodes["end"] > nodes["start"])[::-1]:
        corners = np.arange(nodes["start"][i], nodes["end"][i])
        nodes["start"][i], nodes["end"][i] = at, at + len(corners)
        at += len(corners)
        order.append(corners)
    order = np.concatenate(order)
    turned = (nodes, pos4[order], nrm4[order])
    ctx = api.Context(0)
    rng = np.random.default_rng(5)
    d = np.tile([[0.6, 0.0, 0.8]], (n, 1))
    # into the plane a little behind a grid line, inside the barycentric slack of the triangles before it
    at = np.stack([rng.integers(1, quads, n) / quads + rng.uniform(0, 6e-7, n), rng.uniform(0, 1, n), np.zeros(n)], -1)
    at[::2, 0] = rng.uniform(0, 1, n // 2)  # and anywhere
    o = (at - 0.25 * d).astype(np.float32)
    d = d.astype(np.float32)
    for ascending, arrays in ((True, built), (False, turned)):
        scene = api.Scene(ctx, *arrays)
        by_tree, _ = api.meshmap_routes(ctx, scene, texel_map(ctx, o, d), cull)
        assert by_tree > 0.3 * n if ascending else by_tree == 0
        c1, t1 = mapped(ctx, scene, o, d, cull, api.FLT_MAX)
        c8, t8 = mapped(ctx, scene, o, 8 * d, cull, api.FLT_MAX)
        assert (t1 != api.MISS).mean() > 0.9
        assert np.array_equal(t1, t8) and np.array_equal(bits(c1[:, 1:]), bits(c8[:, 1:]))


@pytest.mark.parametrize("angle,tree", [(None, True), (0.3, True), (1e-2, True), (1e-3, True), (2.6e-4, False),
                                        (2e-4, False)])
def test_route_follows_the_bound(angle, tree):
    """One thin triangle widens the bound of the whole scene: the tree route is
    left where it would meet many more leaves, and where there is no bound."""
    quads = 200
    m = W.grid_plane(quads, heights=0.002 * np.random.default_rng(1).uniform(0, 1, (quads + 1) ** 2))
    if angle is not None:
        nv, e = len(m.positions), 2.0 ** 0.5
        pos = np.concatenate([m.positions, [[0, 0, -0.5], [1, 1, -0.5], [1, 1, -0.5 + e * angle]]])
        m = W.MeshArrays(pos, m.texcoords[:1], [[0, 0, 1]],
                         np.stack([np.arange(nv + 3), np.zeros(nv + 3), np.zeros(nv + 3)], -1),
                         np.concatenate([m.triangles, [[nv, nv + 1, nv + 2]]]))
    ctx = api.Context(0)
    scene = api.Scene.build(ctx, api.Mesh(m))
    n = 1000
    o, d = np.zeros((n, 3)), np.tile([[0.0, 0.0, 1.0]], (n, 1))
    o[:, :2] = np.random.default_rng(2).uniform(0, 1, (n, 2))
    texels, reach = api.meshmap_routes(ctx, scene, texel_map(ctx, o, d), True)
    assert texels > 0.9 * n if tree else texels == 0
    assert reach >= 1.0 and np.isinf(reach) == (angle == 2e-4)
    c1, t1 = mapped(ctx, scene, o, d, True, api.FLT_MAX)
    c8, t8 = mapped(ctx, scene, o, 8 * d, True, api.FLT_MAX)
    assert np.array_equal(t1, t8) and np.array_equal(bits(c1[:, 0]), bits(8 * c8[:, 0]))


@pytest.mark.parametrize("cull", [True, False])
@pytest.mark.parametrize("seed", range(4))
def test_flat_face_outside_its_ancestors_rounded_box(cull, seed):
    """The root's box, rounded from centre and half size, ends an ulp below the
    mesh's flat top: a walk enters it only behind the hit, so a maximum distance
    in between makes the texel a miss."""
    rng = np.random.default_rng(seed)
    f = np.float32
    while True:
        lo, hi = f(-rng.uniform(0.1, 3.0)), f(rng.uniform(0.5, 1.0))
        top = (lo + hi) * f(0.5) + (hi - lo) * f(0.5)
        if top < hi:
            break
    quads, n = 8, 64
    m = W.grid_plane(quads, heights=np.full((quads + 1) ** 2, hi))
    nv = len(m.positions)
    pos = np.concatenate([m.positions, [[0, 0, lo], [1, 0, lo], [0, 1, lo]]]).astype(f)
    verts = np.stack([np.arange(nv + 3), np.zeros(nv + 3), np.zeros(nv + 3)], -1)
    mesh = api.Mesh(W.MeshArrays(pos, m.texcoords[:1], [[0, 0, 1]], verts,
                                 np.concatenate([m.triangles, [[nv, nv + 1, nv + 2]]])))
    ctx = api.Context(0)
    scene = api.Scene.build(ctx, mesh)
    o = np.zeros((n, 3), f)
    o[:, :2] = rng.uniform(0.05, 0.95, (n, 2))
    o[:, 2] = f(1.25) * hi  # both differences below are exact
    d = np.tile([[0, 0, 1]], (n, 1)).astype(f)
    hit, entry = o[0, 2] - hi, o[0, 2] - top
    assert entry > hit
    for max_d, found in ((entry, False), (np.nextafter(entry, f(9)), True), (api.FLT_MAX, True)):
        far = max_d if max_d == api.FLT_MAX else max_d / 8
        c1, t1 = mapped(ctx, scene, o, d, cull, float(max_d))
        c8, t8 = mapped(ctx, scene, o, 8 * d, cull, float(far))
        assert np.array_equal(t1 != api.MISS, np.full(n, found)) and np.array_equal(t1, t8)
        assert np.array_equal(bits(c1[:, 1:]), bits(c8[:, 1:])) and (not found or np.all(c1[:, 0] == hit))
