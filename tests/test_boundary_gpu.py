"""MeshBoundary's face list against a NumPy restatement (unique sorted
corner tuples in lexicographic order, mesh_utils.cpp:98-398): lattice meshes,
a vertex that more boundary faces share than the grouped ordering takes, and
a mesh description whose control point count is too small for its indices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HEX_FACES = ((0, 2, 4, 6), (0, 1, 4, 5), (0, 1, 2, 3), (1, 3, 5, 7), (2, 3, 6, 7), (4, 5, 6, 7))
TET_FACES = ((1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2))   # of corners u, v, w, origin


def corners(shape, p):
    if shape == "hex":
        m = p + 1
        return [p * (i & 1) + m * p * (i >> 1 & 1) + m * m * p * (i >> 2) for i in range(8)]
    nd = (p + 1) * (p + 2) * (p + 3) // 6
    return [p, (p + 1) * (p + 2) // 2 - 1, nd - 1, 0]


def boundary(ctrl_idx, shape, p):
    faces = HEX_FACES if shape == "hex" else TET_FACES
    nd = (p + 1) ** 3 if shape == "hex" else (p + 1) * (p + 2) * (p + 3) // 6
    c = ctrl_idx.reshape(-1, nd)[:, corners(shape, p)]
    seen = {}
    for e in range(len(c)):
        for f, q in enumerate(faces):
            seen.setdefault(tuple(sorted(int(v) for v in c[e, list(q)])), []).append((e, f))
    return np.array([v[0] for _, v in sorted(seen.items()) if len(v) == 1], np.int32)


def fan(n):
    """n tets around one edge (0, 1), closed: vertex 0 and 1 each lie on n
    boundary faces."""
    t = 2 * np.pi * np.arange(n) / n
    xyz = np.concatenate([[[0, 0, -1], [0, 0, 1]],
                          np.stack([np.cos(t), np.sin(t), 0 * t], 1)]).astype(np.float32)
    k = np.arange(n)
    # dofs (0,0,0), u, v, w: origin vertex 0
    idx = np.stack([0 * k, 2 + k, 2 + (k + 1) % n, 0 * k + 1], 1)
    return idx.astype(np.int32).reshape(-1), xyz


@pytest.mark.parametrize("shape,n,p", [("hex", 1, 1), ("hex", 3, 2), ("hex", 9, 1), ("hex", 4, 3),
                                       ("tet", 1, 1), ("tet", 4, 2), ("tet", 3, 3),
                                       ("fan", 100, 1), ("fan", 129, 1), ("fan", 1000, 1)])
@pytest.mark.parametrize("short", [False, True])
def test_boundary_faces_match_restatement(cuda, shape, n, p, short):
    import torch
    from devil_ray_b200 import _lib as L
    from devil_ray_b200 import api, meshgen, render
    if shape == "fan":
        idx, xyz = fan(n)
    elif shape == "hex":
        idx, xyz = meshgen.lattice_ctrl_idx(n, p), meshgen.lattice_points(n, p).astype(np.float32)
    else:
        idx, xyz = meshgen.tet_lattice_ctrl_idx(n, p), meshgen.lattice_points(n, p).astype(np.float32)
    kind = "hex" if shape == "hex" else "tet"
    mesh = api.UnstructuredMesh(idx, xyz, p, device=cuda,
                                shape=L.SHAPE_TENSOR if kind == "hex" else L.SHAPE_SIMPLEX)
    want = boundary(idx, kind, p)
    if short:
        desc = mesh.desc
        mesh.desc = lambda packed=True: _short(desc(packed))
    b = render.MeshBoundary()
    faces, _ = b.execute(mesh)
    torch.cuda.synchronize()
    assert np.array_equal(b.elid_faceid.cpu().numpy(), want)
    assert faces.n_elem == len(want)


def _short(d):
    """A description with half the control points: the face entry point
    does not need them, so its answer is the same."""
    d.n_ctrl = d.n_ctrl // 2
    return d
