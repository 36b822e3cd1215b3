"""The device BVH build's index check."""
import ctypes

import numpy as np
import pytest

from fornos_b200 import _lib as L
from fornos_b200 import api
from fornos_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_index_errors_are_refused():
    """A vertex without a normal (as a PLY file without normals loads) is
    refused before any kernel follows its index, and the context stays usable."""
    ctx = api.Context(0)
    good = W.grid_plane(4)
    bad = good.copy()
    bad.vertices[7, 2] = 0xFFFFFFFF
    for call in (lambda m: api.Scene.build(ctx, m), lambda m: api.BVH.build_flat_device(ctx, m)):
        with pytest.raises(api.FornosError) as e:
            call(api.Mesh(bad))
        assert e.value.code == -1 and "vertex index out of range" in str(e.value)
    assert api.Scene.build(ctx, api.Mesh(good)).info()["corner_count"] == 3 * 32
    ctx.check()


def big():
    return W.grid_plane(400)  # 960k indices: more than one sweep of the check's grid (8 blocks of 256 an SM)


@pytest.mark.parametrize("make", [lambda: W.grid_plane(4), big])
@pytest.mark.parametrize("bad,message", [
    ([("triangles", -1)], "triangle index"), ([("triangles", 0)], "triangle index"),
    ([("positions", -1)], "vertex index"), ([("positions", 0)], "vertex index"),
    ([("normals", -1)], "vertex index"), ([("positions", -1), ("triangles", -1)], "triangle index"),
])
def test_every_index_is_checked(make, bad, message):
    """The first index that does not exist and the largest, in the first and the
    last element; a triangle's error is named before a vertex's.  A mesh's
    creation refuses most of them, so they are written into its arrays after."""
    ctx = api.Context(0)
    arrays = make()
    for beyond in (0, 0xFFFFFFFF):
        mesh = api.Mesh(arrays)
        d = L.MeshDesc()
        assert mesh.lib.fk_mesh_describe(mesh.handle, ctypes.byref(d)) == 0
        tris = np.ctypeslib.as_array(d.triangles, shape=(3 * d.triangle_count,))
        verts = np.ctypeslib.as_array(d.vertices, shape=(3 * d.vertex_count,)).reshape(-1, 3)
        column = {"triangles": (tris, d.vertex_count), "positions": (verts[:, 0], d.position_count),
                  "normals": (verts[:, 2], d.normal_count)}
        for name, at in bad:
            index, count = column[name]
            index[at] = beyond or count
        for call in (api.Scene.build, api.BVH.build_flat_device):
            with pytest.raises(api.FornosError) as e:
                call(ctx, mesh)
            assert e.value.code == -1 and message in str(e.value)
    assert api.Scene.build(ctx, api.Mesh(arrays)).info()["corner_count"] == arrays.triangles.size
    ctx.check()
