"""The device BVH build's index check."""
import pytest

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
