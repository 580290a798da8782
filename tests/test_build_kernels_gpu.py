"""The BVH build's kernels against NumPy restatements at the sizes where
they can go wrong: sub-box splits (orders, partial blocks, degenerate
elements), the radix sort and scan (edges of tiles), the bottom-up tree
(edges of its blocks, runs of equal codes) and the wide tree's two steps.
Everything is compared bit for bit: the steps are defined by 32-bit
operations in a fixed order (data_model/mesh_utils.cpp:482-677,
linear_bvh_builder.cpp:60-397)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


# ------------------------------------------------------------ sub-boxes --

def measure(b):
    e = [F(b[2 * k + 1] - b[2 * k]) for k in range(3)]
    v = F(F(e[0] * e[1]) * e[2])
    if v == 0:
        v = F(F(F(F(2) * e[0]) * e[1]) + F(F(F(2) * e[1]) * e[2]))
        v = F(v + F(F(F(2) * e[2]) * e[0]))
    return v


def hull(q):
    out = np.empty(6, F)
    out[0::2] = np.fmin.reduce(np.vstack([q, np.full((1, 3), np.inf, F)]))
    out[1::2] = np.fmax.reduce(np.vstack([q, np.full((1, 3), -np.inf, F)]))
    return out


def scaled(b):
    out = b.copy()
    for k in range(3):
        lo, hi = b[2 * k], b[2 * k + 1]
        if lo > hi:
            continue
        c = F(F(0.5) * F(lo + hi))
        d = F(F(F(1.000001) * F(0.5)) * F(hi - lo))
        out[2 * k], out[2 * k + 1] = np.fmin(lo, F(c - d)), np.fmax(hi, F(c + d))
    return out


def halves(q, axis, p, dim):
    """De Casteljau at 0.5 along a lattice axis (u fastest): both halves."""
    a = np.moveaxis(q.reshape((p + 1,) * dim + (3,)), dim - 1 - axis, 0)
    rows = [a]
    for _ in range(p):
        r = rows[-1]
        rows.append((r[:-1] * F(0.5) + r[1:] * F(0.5)).astype(F))
    first = np.stack([rows[k][0] for k in range(p + 1)])
    last = np.stack([rows[p - k][k] for k in range(p + 1)])
    back = [np.moveaxis(h, 0, dim - 1 - axis).reshape(-1, 3) for h in (first, last)]
    return back[0], back[1]


def split_element(q, p, dim):
    cps, refs = [q], [np.array([0.0] * dim + [1.0] * dim, F)]
    box = [hull(q)]
    for _ in range(2 * (2 << dim)):
        best, m = 0, measure(box[0])
        for b in range(1, len(box)):
            if measure(box[b]) > m:
                best, m = b, measure(box[b])
        ext = refs[best][dim:] - refs[best][:dim]
        axis = int(np.argmax(ext))
        mid = F(F(refs[best][axis] * F(0.5)) + F(refs[best][dim + axis] * F(0.5)))
        a, b = halves(cps[best], axis, p, dim)
        ra, rb = refs[best].copy(), refs[best].copy()
        ra[dim + axis] = rb[axis] = mid
        cps[best], refs[best], box[best] = a, ra, hull(a)
        cps.append(b), refs.append(rb), box.append(hull(b))
    return np.stack([scaled(b) for b in box]), np.stack(refs)


@pytest.mark.parametrize("dim,p,n", [(3, 1, 1), (3, 1, 5), (3, 2, 3), (3, 2, 4), (3, 3, 2), (3, 3, 9),
                                     (2, 1, 5), (2, 2, 4), (2, 3, 7)])
def test_subboxes_match_restatement(cuda, dim, p, n):
    import torch
    from devil_ray_b200 import api
    rng = np.random.default_rng(100 * dim + 10 * p + n)
    nd = (p + 1) ** dim
    xyz = rng.uniform(-1, 1, (n, nd, 3)).astype(F)
    xyz[0, :, 2] = F(0.25)                     # flat: volume 0, surface area decides
    if n > 1:
        xyz[1] = xyz[1, :1]                    # a point: every measure ties at 0
    if n > 3:
        xyz[3, 0, 0] = np.nan                  # ignored by the hull
        xyz[2, :, 1] = np.nan                  # an empty range in y
    mesh = api.UnstructuredMesh(np.arange(n * nd, dtype=np.int32), xyz.reshape(-1, 3), p, dim=dim,
                                device=cuda)
    got = [t.cpu().numpy() for t in api.elem_subboxes(mesh)]
    torch.cuda.synchronize()
    nb = 33 if dim == 3 else 17
    with np.errstate(invalid="ignore", over="ignore"):
        want = [split_element(xyz[e], p, dim) for e in range(n)]
    assert np.array_equal(got[1], np.repeat(np.arange(n, dtype=np.int32), nb))
    for e in range(n):
        boxes, refs = want[e]
        assert np.array_equal(bits(got[0][e * nb:(e + 1) * nb]), bits(boxes)), f"element {e}"
        assert np.array_equal(bits(got[2][e * nb:(e + 1) * nb]), bits(refs)), f"element {e}"


# ------------------------------------------------------- sort and scan --

# tiles of 1024 keys below one tile of 4096 an SM, of 4096 above
@pytest.mark.parametrize("n", [1, 31, 511, 1023, 1024, 1025, 4095, 4096, 4097, 3 * 4096 + 7, 300001,
                               200 * 4096, 200 * 4096 + 1, 250 * 4096 - 5])
@pytest.mark.parametrize("bits_", [1, 8, 9, 30, 32])
def test_radix_sort_is_stable_at_tile_edges(cuda, n, bits_):
    import torch
    from devil_ray_b200 import api
    rng = np.random.default_rng(n + bits_)
    keys = rng.integers(0, 1 << bits_, n, dtype=np.uint64).astype(np.uint32)
    if n > 600:
        keys[100:n // 2] = keys[100]           # a long run of one digit
    k, v = api.radix_sort_pairs(torch.as_tensor(keys.view(np.int32), device=cuda),
                                torch.arange(n, dtype=torch.int32, device=cuda), bits_)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(v.cpu().numpy(), order)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 9 * 4096 + 1])
def test_compaction_at_scan_tile_edges(cuda, n):
    """cull_rays compacts by the exclusive scan: rays that miss a box."""
    import torch
    from devil_ray_b200 import render
    rng = np.random.default_rng(n)
    hit = rng.random(n) < 0.6
    rays = np.zeros((n, 9), F)
    rays[:, 2] = 1.0                            # along z
    rays[:, 4] = np.where(hit, 0.5, 3.0)
    rays[:, 5], rays[:, 6], rays[:, 7] = 0.5, -2.0, np.inf
    rays[:, 8] = np.arange(n, dtype=np.int32).view(F)
    out = render.cull_rays(torch.as_tensor(rays, device=cuda), [0, 1, 0, 1, 0, 1])
    assert np.array_equal(out.cpu().numpy()[:, 8].view(np.int32), np.flatnonzero(hit))


# ---------------------------------------------------------------- trees --

def delta(codes):
    """Common prefix of neighbouring codes, the index breaking ties
    (linear_bvh_builder.cpp:149-167)."""
    out = np.empty(len(codes) - 1, int)
    for j in range(len(codes) - 1):
        x = int(codes[j]) ^ int(codes[j + 1])
        out[j] = 32 - x.bit_length() if x else 64 - (j ^ (j + 1)).bit_length()
    return out


def radix_tree(codes, boxes):
    """Node records of the Karras tree, by recursion over the split with the
    shortest prefix; boxes: sorted leaf boxes x0 x1 y0 y1 z0 z1."""
    n = len(codes)
    d = delta(codes)
    rec = np.zeros((n - 1, 16), F)
    kids = rec.view(np.int32)

    def visit(l, r, left):
        """(child code, box) of the node over [l, r], a left child or not."""
        if l == r:
            return -(l + 1), boxes[l]
        me = 0 if (l, r) == (0, n - 1) else (r if left else l)
        p = l + int(np.argmin(d[l:r]))
        (cl, bl), (cr, br) = visit(l, p, True), visit(p + 1, r, False)
        rec[me, :12] = np.concatenate([bl[0::2], bl[1::2], br[0::2], br[1::2]])
        kids[me, 12], kids[me, 13] = cl, cr
        u = np.empty(6, F)
        u[0::2], u[1::2] = np.fmin(bl[0::2], br[0::2]), np.fmax(bl[1::2], br[1::2])
        return 4 * me, u

    visit(0, n - 1, False)
    return rec


def _tree_mesh(kind, n_elem, cuda):
    from devil_ray_b200 import api
    rng = np.random.default_rng(n_elem)
    if kind == "scattered":
        xyz = rng.uniform(0, 1, (n_elem, 1, 3)) + 0.1 * rng.uniform(0, 1, (n_elem, 8, 3))
        idx = np.arange(8 * n_elem)
    elif kind == "repeated":  # one element n times: every code occurs n times
        xyz, idx = rng.uniform(0, 1, (1, 8, 3)), np.tile(np.arange(8), n_elem)
    else:                     # points in one place: all codes equal
        xyz, idx = np.full((1, 8, 3), 0.5), np.tile(np.arange(8), n_elem)
    return api.UnstructuredMesh(idx.astype(np.int32), xyz.reshape(-1, 3).astype(F), 1, device=cuda)


# 33 leaves an element; the tree's blocks hold 256 leaves
@pytest.mark.parametrize("kind,n_elem", [("scattered", 1), ("scattered", 7), ("scattered", 8),
                                         ("scattered", 31), ("scattered", 256), ("repeated", 8),
                                         ("repeated", 70), ("point", 1), ("point", 40)])
def test_bottom_up_tree_matches_top_down(cuda, kind, n_elem):
    import sys
    import torch
    from devil_ray_b200 import api
    mesh = _tree_mesh(kind, n_elem, cuda)
    b = mesh.build_bvh(keep_codes=True)
    aabbs, _, refs, bounds = api.elem_subboxes(mesh)
    codes = api.morton_codes(aabbs, bounds).cpu().numpy().view(np.uint32)
    torch.cuda.synchronize()
    order = np.argsort(codes, kind="stable")
    assert np.array_equal(b.sorted_codes.cpu().numpy().view(np.uint32), codes[order])
    assert np.array_equal(b.aabb_ids.cpu().numpy(), order)
    assert np.array_equal(b.leaf_nodes.cpu().numpy(), order // 33)
    sys.setrecursionlimit(20000)
    want = radix_tree(codes[order], aabbs.cpu().numpy()[order])
    assert np.array_equal(bits(b.inner_nodes.cpu().numpy()), bits(want))


def collapse(nodes):
    """4-wide collapse of the binary records: even-depth nodes in index
    order, their grandchildren (children where those are leaves)."""
    kids = nodes.view(np.int32)[:, 12:14]
    depth = np.zeros(len(nodes), int)
    stack = [0]
    while stack:
        i = stack.pop()
        for c in kids[i]:
            if c >= 0:
                depth[c // 4] = depth[i] + 1
                stack.append(c // 4)
    wide_of = np.cumsum(depth % 2 == 0) - 1
    out = []
    for i in np.flatnonzero(depth % 2 == 0):
        got = []
        for side, c in enumerate(kids[i]):
            if c < 0:
                got.append((nodes[i, 6 * side:6 * side + 6], c))
                continue
            for s2, g in enumerate(kids[c // 4]):
                got.append((nodes[c // 4, 6 * s2:6 * s2 + 6], g if g < 0 else wide_of[g // 4]))
        row = np.zeros(32, F)
        code = row.view(np.int32)
        for k in range(4):
            box, c = got[k] if k < len(got) else (np.array([np.inf] * 3 + [-np.inf] * 3, F), -2**31)
            row[k:24:4], code[24 + k] = box, c
        code[28] = len(got)
        out.append(row)
    return np.stack(out), int(depth.max()) // 2 + 1


# the depth pass takes 1024 nodes a block, the emit pass 128
@pytest.mark.parametrize("kind,n_elem", [("scattered", 1), ("scattered", 4), ("scattered", 31),
                                         ("scattered", 32), ("scattered", 200), ("repeated", 70),
                                         ("point", 100)])
def test_wide_plan_and_emit(cuda, kind, n_elem):
    import torch
    from devil_ray_b200 import _lib as L
    b = _tree_mesh(kind, n_elem, cuda).build_bvh()
    want, depth = collapse(b.inner_nodes.cpu().numpy())
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for shift in (0, 1):                        # ids on and off a 16-byte boundary
        ids = torch.full((b.n_inner + shift,), -7, dtype=torch.int32, device=cuda)[shift:]
        d = b.desc()
        assert L.lib().drb_bvh_widen_plan(C.byref(d), C.c_void_p(ids.data_ptr()), s) == 0
        assert (d.n_wide, d.wide_depth) == (len(want), depth)
        out = torch.empty((d.n_wide, 32), dtype=torch.float32, device=cuda)
        assert L.lib().drb_bvh_widen_emit(C.byref(d), C.c_void_p(ids.data_ptr()),
                                          C.c_void_p(out.data_ptr()), d.n_wide - 1, s) != 0
        assert L.lib().drb_bvh_widen_emit(C.byref(d), C.c_void_p(ids.data_ptr()),
                                          C.c_void_p(out.data_ptr()), d.n_wide, s) == 0
        assert np.array_equal(bits(out.cpu().numpy()), bits(want))
    b.widen()
    assert np.array_equal(bits(b.wide_nodes.cpu().numpy()), bits(want))


def test_widen_allocates_on_its_stream(cuda, monkeypatch):
    """What widen(stream) writes on a stream is that stream's memory, not a
    block that work queued on the current stream may still use."""
    import torch
    from devil_ray_b200 import api
    b = _tree_mesh("scattered", 31, cuda).build_bvh()
    want = b.widen().wide_nodes.cpu().numpy()
    side = torch.cuda.Stream(cuda)
    torch.cuda.synchronize()
    empty, made_on = torch.empty, []

    def recorded(*args, **kw):
        made_on.append(torch.cuda.current_stream(cuda))
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", recorded)
    b.widen(side)
    monkeypatch.undo()
    assert made_on and all(s == side for s in made_on)
    assert torch.cuda.current_stream(cuda) != side
    torch.cuda.synchronize()
    assert np.array_equal(bits(b.wide_nodes.cpu().numpy()), bits(want))


# scales: lists of a few leaves, of some tens, of about a hundred (more than
# 64 comparisons an entry: radix passes), and one cell with every leaf (more
# than 32 leaves a cell: radix passes at once).  power: control points raised
# to it, so that leaves crowd into the cells at one corner, at 264,000 leaves
# so many that a sixteenth of them shows it
@pytest.mark.parametrize("n,scale,power", [(3, 0.4, 1), (5, 1.0, 1), (9, 2.6, 1), (9, 5.0, 1),
                                           (4, 1e6, 1), (9, 1.0, 4), (20, 1.0, 6), (20, 1.0, 1), (20, 1.5, 1.5)])
def test_grid_lists_of_every_length(cuda, n, scale, power):
    import torch
    from devil_ray_b200 import api, meshgen
    m = meshgen.trilinear_distorted_mesh(n, 2, 0.15, seed=11)
    xyz = m.xyz if power == 1 else np.clip(m.xyz, 0, 1) ** np.float32(power)
    g = api.UnstructuredMesh(m.ctrl_idx, xyz, m.order, device=cuda)
    b = g.get_bvh().build_grid(scale)
    torch.cuda.synchronize()
    dims, origin, inv = b.grid_geom
    box = b.grid_boxes.cpu().numpy()
    lo, hi = box[:, :3], box[:, 4:7]

    def axis(x, d):
        v = (x - np.float32(origin[d])).astype(np.float32) * np.float32(inv[d])
        return np.floor(np.clip(v, np.float32(0), np.float32(dims[d] - 1))).astype(np.int64)

    c0 = np.stack([axis(lo[:, d], d) for d in range(3)], 1)
    span = np.stack([axis(hi[:, d], d) for d in range(3)], 1) - c0 + 1
    count = span.prod(1)
    leaf = np.repeat(np.arange(b.n_leaf), count)
    i = np.arange(leaf.size) - np.repeat(np.cumsum(count) - count, count)
    s, c = span[leaf], c0[leaf]
    x, y, z = c[:, 0] + i % s[:, 0], c[:, 1] + i // s[:, 0] % s[:, 1], c[:, 2] + i // (s[:, 0] * s[:, 1])
    cell = (z * dims[1] + y) * dims[0] + x
    order = np.lexsort((leaf, cell))
    n_cells = dims[0] * dims[1] * dims[2]
    start = np.searchsorted(cell[order], np.arange(n_cells + 1))
    assert np.array_equal(b.grid_start.cpu().numpy(), start)
    assert np.array_equal(b.grid_entries.cpu().numpy(), leaf[order])


def test_grid_lists_just_below_the_entry_limit(cuda):
    """2^31 - 2 entries, the largest count below the limit that rows of
    equal lists make: 9,513 rows of 3,641 cells, 62 leaves a row.  Entry
    indices run past what a signed index plus one warp holds.  (17 GB.)"""
    import torch
    from devil_ray_b200 import _lib as L
    dims, per_row = (3641, 151, 63), 62
    rows = dims[1] * dims[2]
    n_cells, n = rows * dims[0], rows * per_row
    m = n_cells * per_row
    assert m == 2**31 - 2
    if torch.cuda.mem_get_info(cuda)[0] < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    # node records that hold two leaves each (the others hold none)
    row = torch.arange(n, device=cuda) // per_row
    y, z = (row % dims[1]).float(), (row // dims[1]).float()
    lo = torch.stack([torch.full_like(y, 0.5), y + 0.25, z + 0.25], 1)
    hi = torch.stack([torch.full_like(y, dims[0] - 0.5), y + 0.75, z + 0.75], 1)
    rec = torch.zeros((n - 1, 16), dtype=torch.float32, device=cuda)
    rec[:n // 2, :12] = torch.cat([lo, hi], 1).reshape(n // 2, 12)
    rec.view(torch.int32)[:n // 2, 12:14] = -1 - torch.arange(n, dtype=torch.int32,
                                                             device=cuda).reshape(-1, 2)
    leaf_nodes = torch.arange(n, dtype=torch.int32, device=cuda)
    start = torch.empty(n_cells + 1, dtype=torch.int32, device=cuda)
    entries = torch.full((m,), -1, dtype=torch.int32, device=cuda)
    boxes = torch.empty((n, 8), dtype=torch.float32, device=cuda)
    d = L.DrbBvh()
    d.n_inner, d.n_leaf = n - 1, n
    d.inner_nodes, d.leaf_nodes = rec.data_ptr(), leaf_nodes.data_ptr()
    d.grid_start, d.grid_entries, d.grid_boxes = (t.data_ptr() for t in (start, entries, boxes))
    for q in range(3):
        d.grid_dims[q], d.grid_origin[q], d.grid_inv[q] = dims[q], 0.0, 1.0
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L.check(L.lib().drb_bvh_grid_build(C.byref(d), s), "drb_bvh_grid_build")
    want = per_row * torch.arange(n_cells + 1, dtype=torch.int64, device=cuda)
    assert torch.equal(start.long(), want)
    del want
    lists = entries.reshape(rows, dims[0], per_row)
    leaves = torch.arange(n, dtype=torch.int32, device=cuda).reshape(rows, 1, per_row)
    for r in range(0, rows, 500):
        assert torch.equal(lists[r:r + 500],
                           leaves[r:r + 500].expand(-1, dims[0], -1)), f"row {r}"
    del entries, lists
    torch.cuda.empty_cache()
