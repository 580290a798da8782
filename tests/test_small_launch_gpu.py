"""The launch shape for few queries against the one for many: the same queries
give the same bits."""
import pytest

from devil_ray_b200 import _lib as L
from devil_ray_b200 import api, meshgen

pytestmark = pytest.mark.gpu


def _mesh(kind, n, p):
    if kind == "tet":
        return meshgen.tet_warped_mesh(n, p, 0.05, jitter=0.01, seed=5), L.SHAPE_SIMPLEX
    return meshgen.warped_mesh(n, p, 0.08, jitter=0.01, seed=5), L.SHAPE_TENSOR


# one query; a warp's chunk and its edges; one more chunk than warps; the
# largest small batch and one above it
@pytest.mark.parametrize("count", [1, 31, 33, 2368, 2369, 75777, 103600, 103601])
@pytest.mark.parametrize("kind,p,lists", [("hex", 2, "grid"), ("hex", 3, "tree"), ("tet", 2, "tree")])
def test_small_batch_equals_ordered(cuda, kind, p, lists, count):
    import torch
    m, shape = _mesh(kind, 5, p)
    g = api.UnstructuredMesh(m.ctrl_idx, m.xyz, m.order, device=cuda, shape=shape)
    bvh = g.get_bvh()
    if lists == "grid":
        bvh.build_grid(0.75)
    loc = api.BatchedLocator(g, tol=1e-5, max_steps=20, bvh=bvh)
    q = torch.as_tensor(meshgen.uniform_queries(count, 3), device=cuda)
    order = torch.arange(count, dtype=torch.int32, device=cuda).flip(0).contiguous()
    for a, b in zip(loc.locate(q, stats=True), loc.locate(q, order=order, stats=True)):
        assert torch.equal(a, b)
