"""One Newton step on elements whose Jacobian is diagonal and whose values at
the first guess are exact in 32 bits: the step is then the rounded quotient of
the residual and the extent, added to the guess, so every bit of the result is
known (newton_solver.hpp:33-74, matrix.hpp:221-373).  A product with a rounded
reciprocal differs in the last bit for a share of the queries, and is not
finite for extents below 2^-128."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32
# halves and thirds exact: the control points of orders 1 to 3 are too
EXTENT = np.array([3.0, 9.0, 21.0], F)


def _box(p, dim=3):
    """Control points of one axis-aligned box (x fastest) from the origin."""
    t = np.arange(p + 1, dtype=F) / F(p)
    if dim == 2:
        y, x = np.meshgrid(t, t, indexing="ij")
        return np.stack([x, y, 0 * x], -1).reshape(-1, 3) * EXTENT * np.array([1, 1, 0], F)
    z, y, x = np.meshgrid(t, t, t, indexing="ij")
    # t * extent rounds to the exact k * extent / p
    return (np.stack([x, y, z], -1).reshape(-1, 3) * EXTENT).astype(F)


def _step(q, guess, extent):
    return F(guess) + (q - F(guess) * extent) / extent


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("exponent", [0, -130])
def test_hex_step_is_the_rounded_quotient(cuda, p, exponent):
    import torch
    from devil_ray_b200 import api, learned
    scale = np.ldexp(F(1), exponent).astype(F)
    xyz = _box(p) * scale
    assert np.array_equal(np.ldexp(xyz.astype(np.float64), -exponent), _box(p).astype(np.float64))
    mesh = api.UnstructuredMesh(np.arange(len(xyz), dtype=np.int32), xyz, p, device=cuda)
    n = 4096
    q = (np.random.default_rng(p).uniform(0, 1, (n, 3)).astype(F) * EXTENT * scale).astype(F)
    pts = torch.as_tensor(q, device=cuda)
    elem = torch.zeros(n, dtype=torch.int32, device=cuda)
    ref, found, _ = learned.newton_pairs(mesh, elem, pts, tol=10.0, max_steps=1)
    want = _step(q, 0.5, EXTENT * scale)
    assert np.array_equal(ref.cpu().numpy().view(np.int32), want.view(np.int32))
    assert bool((found != 0).all())


@pytest.mark.parametrize("kind,p", [("hex", 1), ("hex", 2), ("hex", 3), ("tet", 1), ("quad", 1),
                                    ("quad", 2)])
@pytest.mark.parametrize("batched", [False, True])
def test_located_step_is_the_rounded_quotient(cuda, kind, p, batched):
    from devil_ray_b200 import _lib as L
    from devil_ray_b200 import api
    rng = np.random.default_rng(10 + p)
    n = 4096
    u = rng.uniform(0, 1, (n, 3))
    if kind == "tet":
        xyz = np.concatenate([np.zeros((1, 3), F), np.diag(EXTENT)])    # origin, u, v, w
        u = rng.dirichlet([1, 1, 1, 1], n)[:, :3]
        mesh = api.UnstructuredMesh(np.arange(4, dtype=np.int32), xyz, p, device=cuda,
                                    shape=L.SHAPE_SIMPLEX)
    else:
        xyz = _box(p, 2 if kind == "quad" else 3)
        mesh = api.UnstructuredMesh(np.arange(len(xyz), dtype=np.int32), xyz, p, device=cuda,
                                    dim=2 if kind == "quad" else 3)
    q = (u.astype(F) * EXTENT).astype(F)
    dims = 3
    if kind == "quad":
        q[:, 2] = 0
        dims = 2
    if batched:
        loc = api.BatchedLocator(mesh, tol=10.0, max_steps=1, guess_mode=L.GUESS_ELEM_CENTER)
        cell, ref = loc.locate(q)
    else:
        cell, ref = mesh.locate(q, tol=10.0, max_steps=1, guess_mode=L.GUESS_ELEM_CENTER)
    hit = cell.cpu().numpy() == 0
    assert hit.mean() > 0.99
    want = _step(q[:, :dims], 0.25 if kind == "tet" else 0.5, EXTENT[:dims])
    got = ref.cpu().numpy()[:, :dims]
    assert np.array_equal(got[hit].view(np.int32), want[hit].view(np.int32))
