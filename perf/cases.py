"""Performance cases of the library: what its users have it do, through its
public entry points, with 64-bit restatements of the computed results.

Kinds of case (sizes are those of the test and benchmark meshes, and smaller
and larger ones of the same families):

  probe     PointLocation.execute: field values at a handful of points.  An
            interactive probe or a simulation's tracer points; launches and
            host work count.
  locate    BatchedLocator.locate at tolerance 1e-5: point location over the
            traversal tree or over the grid candidate lists, hexes and tets.
  learned   LearnedLocator.locate: first candidates, network guess, locate.
  setup     A new mesh, as each time step of a moving mesh brings one: packed
            rows, the BVH with its traversal tree, and (lists "grid") the
            leaf maps and grid candidate lists of the batched locate.
  boundary  MeshBoundary.execute and the BVH of its faces.
  surface   Surface.render: one frame of the boundary, rays to framebuffer.
  volume    Volume.render: one frame, plain march (march 0, the default) or
            coherent march (1, 2), lit or not.
  train     One training step of the guess network on a batch: features,
            loss and gradients, Adam update.

All meshes fill [0,1]^3; their boundary control points keep the lattice
position on the boundary.
"""
import itertools
import math

import torch

from devil_ray_b200 import _lib as L
from devil_ray_b200 import api, learned, meshgen, render

DEVICE = "cuda"


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # a probe of a small mesh at a thousand points, two fields
        {"name": "probe_1k", "kind": "probe", "cells": "hex", "n": 16, "p": 2, "points": 1000},
        # a tracer batch over an order-3 mesh, traversal tree
        {"name": "locate_tree_1m", "kind": "locate", "cells": "hex", "n": 32, "p": 3,
         "points": 1000003, "lists": "tree", "guess": "linear"},
        # the batched point location workload at its full size, grid lists
        {"name": "locate_grid_16m", "kind": "locate", "cells": "hex", "n": 64, "p": 2,
         "points": 16777216, "lists": "grid", "guess": "linear"},
        # the tet workload, a quarter of its queries
        {"name": "locate_tet_4m", "kind": "locate", "cells": "tet", "n": 32, "p": 2,
         "points": 4194304, "lists": "tree", "guess": "centre"},
        # the learned-guess workload, a quarter of its queries
        {"name": "learned_4m", "kind": "learned", "n": 64, "p": 2, "points": 4194304,
         "lists": "grid"},
        # an ordinary order-3 mesh made ready for rendering or location
        {"name": "setup_p3_32", "kind": "setup", "cells": "hex", "n": 32, "p": 3, "lists": "tree"},
        # the point location workload's mesh made ready, leaf maps and grid lists too
        {"name": "setup_p2_64_grid", "kind": "setup", "cells": "hex", "n": 64, "p": 2,
         "lists": "grid"},
        # the boundary of that mesh made ready for surface rendering
        {"name": "boundary_p2_64", "kind": "boundary", "cells": "hex", "n": 64, "p": 2},
        # the surface workload's frame
        {"name": "surface_p3_1024", "kind": "surface", "cells": "hex", "n": 32, "p": 3,
         "width": 1024, "lit": True},
        # the small volume workload's frame with the renderer's defaults
        {"name": "volume_p2_256", "kind": "volume", "cells": "hex", "n": 8, "p": 2, "width": 256,
         "samples": 500, "march": 0, "lit": True},
        # a large frame of an order-3 mesh, coherent march
        {"name": "volume_p3_1024", "kind": "volume", "cells": "hex", "n": 64, "p": 3,
         "width": 1024, "samples": 1000, "march": 2, "lit": True},
        # one step of the guess network's training
        {"name": "train_16k", "kind": "train", "n": 32, "p": 2, "batch": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds' ranges: orders 1 to 3, hexes and tets,
    meshes from 3 elements an axis to the listed sizes, from one query to
    millions, frames from 33 to 1024 pixels wide."""
    kind = rng.choice(["probe", "locate", "locate", "learned", "setup", "setup", "boundary",
                       "surface", "volume", "volume", "train"])
    p = rng.choice([1, 2, 3])
    cells = rng.choice(["hex", "hex", "tet"])
    top = {1: 48, 2: 40, 3: 32}[p] if cells == "hex" else {1: 24, 2: 20, 3: 14}[p]
    n = _log_int(rng, 3, top)
    if kind == "probe":
        return {"kind": kind, "cells": cells, "n": min(n, 24), "p": p,
                "points": _log_int(rng, 1, 100000)}
    if kind == "locate":
        return {"kind": kind, "cells": cells, "n": n, "p": p, "points": _log_int(rng, 300, 2000000),
                "lists": rng.choice(["tree", "grid"]) if cells == "hex" else "tree",
                "guess": rng.choice(["linear", "centre", "subref"])}
    if kind == "learned":
        return {"kind": kind, "n": _log_int(rng, 6, 40), "p": p,
                "points": _log_int(rng, 1000, 1500000), "lists": rng.choice(["tree", "grid"])}
    if kind == "setup":
        return {"kind": kind, "cells": cells, "n": n, "p": p,
                "lists": rng.choice(["tree", "grid"]) if cells == "hex" else "tree"}
    if kind == "boundary":
        return {"kind": kind, "cells": cells, "n": n, "p": p}
    if kind == "surface":
        return {"kind": kind, "cells": cells, "n": n, "p": p, "width": _log_int(rng, 33, 1024),
                "lit": rng.random() < 0.7}
    if kind == "volume":
        return {"kind": kind, "cells": cells, "n": min(n, 24), "p": p,
                "width": _log_int(rng, 33, 512), "samples": _log_int(rng, 50, 500),
                "march": rng.choice([0, 1, 2]), "lit": rng.random() < 0.7}
    return {"kind": kind, "n": min(n, 32), "p": p, "batch": 128 * _log_int(rng, 1, 512)}


# ----------------------------------------------------------------- inputs --

def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _uniform(shape, lo, hi, gen):
    return torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float64) * (hi - lo) + lo


def _ctrl_idx(cells, n, p):
    idx = meshgen.lattice_ctrl_idx(n, p) if cells == "hex" else meshgen.tet_lattice_ctrl_idx(n, p)
    return torch.as_tensor(idx, device=DEVICE)


def _warped_points(n, p, amp, jitter, gen):
    """Lattice points of [0,1]^3, interior ones displaced by a smooth warp
    and a uniform jitter (float32 [m^3, 3], x fastest)."""
    m = p * n + 1
    t = torch.linspace(0.0, 1.0, m, device=DEVICE, dtype=torch.float64)
    Z, Y, X = torch.meshgrid(t, t, t, indexing="ij")
    xyz = torch.stack([X, Y, Z], dim=-1)
    s = torch.sin(2 * math.pi * t)
    d = amp * s[:, None, None] * s[None, :, None] * s[None, None, :]
    move = d[..., None] + _uniform((m, m, m, 3), -jitter, jitter, gen)
    xyz[1:-1, 1:-1, 1:-1] += move[1:-1, 1:-1, 1:-1]
    return xyz.reshape(-1, 3).float()


def _trilinear_points(n, p, distortion, gen):
    """Vertex lattice displaced by up to distortion x h (boundary vertices
    stay on the boundary); the order-p control points interpolate the
    corners, so every element is a trilinear map."""
    t = torch.linspace(0.0, 1.0, n + 1, device=DEVICE, dtype=torch.float64)
    Z, Y, X = torch.meshgrid(t, t, t, indexing="ij")
    v = torch.stack([X, Y, Z], dim=-1)
    d = _uniform((n + 1, n + 1, n + 1, 3), -distortion / n, distortion / n, gen)
    for axis in range(3):           # component `axis` belongs to dimension 2 - axis
        for end in (0, n):
            d.select(2 - axis, end)[..., axis] = 0.0
    v = v + d
    for dim in range(3):
        parts = []
        a0 = v.narrow(dim, 0, n)
        a1 = v.narrow(dim, 1, n)
        for a in range(p):
            parts.append(a0 * (1 - a / p) + a1 * (a / p))
        w = torch.stack(parts, dim=dim + 1).flatten(dim, dim + 1)
        v = torch.cat([w, v.narrow(dim, n, 1)], dim=dim)
    return v.reshape(-1, 3).float()


def _points(case, gen):
    """Control points of a case's mesh, by kind as its workload has them."""
    n, p = case["n"], case["p"]
    cells = case.get("cells", "hex")
    if case["kind"] in ("locate", "learned", "setup", "train") and cells == "hex" and p < 3:
        return _trilinear_points(n, p, 0.15, gen)
    jitter = min(0.01, 0.1 / (p * n))
    return _warped_points(n, p, 0.05, jitter, gen)


def _fields(xyz, seed):
    """Two scalar fields; the seed moves the first one's phase."""
    x, y, z = (xyz[:, k].double() for k in range(3))
    a, b = ((seed * q) % 1.0 - 0.5 for q in (0.618034, 0.754878))
    f = torch.sin(3.0 * x + a) * torch.cos(2.0 * y + b) + z * z
    blob = torch.exp(-((x - 0.4) ** 2 + (y - 0.6) ** 2 + (z - 0.5) ** 2) / 0.08)
    return f.float(), blob.float()


def _queries(count, gen):
    """Uniform in a cube padded so that 8 % of the queries lie outside."""
    pad = meshgen.QUERY_PAD
    return _uniform((count, 3), -pad, 1.0 + pad, gen).float()


def _scene(case, seed, gen):
    """Control points and connectivity of a case's mesh.  The sizes of the
    trees and lists that setup and boundary return depend on the geometry,
    so there the seed keeps it up to a power of two (another unit) and
    renumbers the elements, starting at another one."""
    n, p, cells = case["n"], case["p"], case.get("cells", "hex")
    idx = _ctrl_idx(cells, n, p)
    if case["kind"] not in ("setup", "boundary"):
        return _points(case, gen), idx
    xyz = _points(case, _gen(1)) * 2.0 ** (seed % 7 - 3)
    elems, nd, _ = _sizes(case)
    return xyz, torch.roll(idx.view(elems, nd), seed % elems, 0).reshape(-1)


def _shape(case):
    return L.SHAPE_TENSOR if case.get("cells", "hex") == "hex" else L.SHAPE_SIMPLEX


GUESS = {"linear": L.GUESS_SUBBOX_LINEAR, "centre": L.GUESS_ELEM_CENTER,
         "subref": L.GUESS_SUBREF_CENTER}


def _camera(width):
    c = meshgen.CAMERA
    return render.Camera(width, width, c["pos"], c["look_at"], c["up"], c["fov"])


def _color_table():
    t = render.ColorTable()
    for pos, *rgb in meshgen.TF_RGB:
        t.add_point(pos, rgb)
    return t


def _identity_network(order, gen):
    """Parameters of a network that returns the point's place in the
    element's control-point box, 0.5 + 0.5 x, with small random weights
    elsewhere: gelu(a) - gelu(-a) = a, so pairs of hidden units carry each
    coordinate through both layers.  What a trained network of the workload
    is close to, and the same for every build of the library."""
    lay = learned.Layout(order)
    w = (torch.rand(lay.n_params, generator=gen, device=DEVICE) - 0.5) * 0.02
    w1 = w[lay.W1:lay.B1].view(learned.N_HID, lay.n_in)
    w2 = w[lay.W2:lay.B2].view(learned.N_HID, learned.N_HID)
    w3 = w[lay.W3:lay.B3].view(learned.N_OUT, learned.N_HID)
    w1[:6], w2[:6], w3[:, :6] = 0.0, 0.0, 0.0
    w2[6:], w3[:, 6:] = w2[6:] * 0.1, w3[:, 6:] * 0.1
    for k in range(3):
        for s, sign in enumerate((1.0, -1.0)):
            w1[2 * k + s, lay.n_in - 3 + k] = sign
            w2[2 * k + s, 2 * k], w2[2 * k + s, 2 * k + 1] = sign, -sign
            w3[k, 2 * k + s] = 0.5 * sign
    w[lay.B1:lay.W2], w[lay.B2:lay.W3], w[lay.B3:] = 0.0, 0.0, 0.5
    return w


def _network(order, params):
    model = learned.GuessMLP(DEVICE, 0, order)
    model.params.copy_(params)
    model.prepare()
    return model


def _pairs(case, gen):
    """A training batch: elements, reference points mapped forward (64-bit,
    then rounded), the reference points as labels, a few rejected pairs."""
    n, p, b = case["n"], case["p"], case["batch"]
    xyz = _points(case, gen)
    idx = _ctrl_idx("hex", n, p)
    elem = torch.randint(0, n ** 3, (b,), generator=gen, device=DEVICE, dtype=torch.int32)
    r = _uniform((b, 3), 0.0, 1.0, gen)
    nd = (p + 1) ** 3
    cps = xyz.double()[idx.view(-1, nd)[elem.long()].long()]
    pts = _hex_eval(cps, r, p)[0].float()
    weight = (torch.rand(b, generator=gen, device=DEVICE) > 0.01).float()
    return xyz, idx, elem, pts, r.float(), weight


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    n, p = case["n"], case["p"]
    if kind == "train":
        xyz, idx, elem, pts, label, weight = _pairs(case, gen)
        model = _network(p, _identity_network(p, gen))
        return {"case": case, "mesh": api.UnstructuredMesh(idx, xyz, p, device=DEVICE),
                "model": model, "elem": elem, "pts": pts, "label": label, "weight": weight,
                "ws": model.workspace(case["batch"])}
    xyz, idx = _scene(case, seed, gen)
    shape = _shape(case)
    if kind == "setup":
        return {"case": case, "xyz": xyz, "idx": idx, "shape": shape}
    mesh = api.UnstructuredMesh(idx, xyz, p, device=DEVICE, shape=shape)
    state = {"case": case, "mesh": mesh}
    if kind in ("probe", "boundary", "surface", "volume"):
        names = ("wave", "blob")
        fields = {k: render.UnstructuredField(idx, v, p, name=k, device=DEVICE, shape=shape)
                  for k, v in zip(names, _fields(xyz, seed))}
        state["fields"] = fields
    if kind == "probe":
        state["points"] = _queries(case["points"], gen)
        mesh.get_bvh()
        q = render.PointLocation()
        for k in state["fields"]:
            q.add_var(k)
        q.empty_val(-2.0)
        state["query"] = q
    elif kind == "locate":
        state["points"] = _queries(case["points"], gen)
        bvh = mesh.get_bvh()
        config = None
        if case["guess"] == "linear":
            bvh.build_leaf_maps(mesh)
        if case["lists"] == "grid":
            bvh.build_grid(0.75)
            config = L.DrbLocateConfig(128, 0, 64, 2, 0)
        state["locator"] = api.BatchedLocator(mesh, 1e-5, 20, GUESS[case["guess"]], config)
    elif kind == "learned":
        state["points"] = _queries(case["points"], gen)
        bvh = mesh.get_bvh()
        if case["lists"] == "grid":
            bvh.build_grid(0.75)
        model = _network(p, _identity_network(p, gen))
        state["locator"] = learned.LearnedLocator(mesh, model, 1e-5, 20, None, bvh)
    elif kind == "surface":
        faces, face_field = render.MeshBoundary().execute(mesh, state["fields"]["wave"])
        surface = render.Surface(faces, face_field)
        surface.color_map().color_table(_color_table())
        faces.get_bvh()
        face_field.range()
        state["surface"], state["camera"] = surface, _camera(case["width"])
        del state["mesh"], state["fields"]
    elif kind == "volume":
        vol = render.Volume(mesh, state["fields"]["wave"])
        table = _color_table()
        for pos, a in meshgen.TF_ALPHA:
            table.add_alpha(pos, a)
        vol.color_map().color_table(table)
        vol.samples(case["samples"])
        vol.use_lighting(case["lit"])
        vol.coherent = case["march"]
        mesh.get_bvh()
        state["fields"]["wave"].range()
        state["volume"], state["camera"] = vol, _camera(case["width"])
    return state


# -------------------------------------------------------------------- run --

def _bits(t):
    return t.view(torch.int32)


def _mesh_outputs(mesh, bvh):
    """The mesh's and its BVH's arrays; node records as integers, which also
    compares the child codes they hold."""
    return {"packed": mesh.packed, "inner": _bits(bvh.inner_nodes), "wide": _bits(bvh.wide_nodes),
            "leaf": bvh.leaf_nodes, "ids": bvh.aabb_ids, "ref": bvh.ref_boxes,
            "bounds": bvh.bounds}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "probe":
        return state["query"].execute(state["mesh"], state["fields"], state["points"])
    if kind in ("locate", "learned"):
        cell, ref = state["locator"].locate(state["points"])
        return {"cell": cell, "ref": ref}
    if kind == "setup":
        mesh = api.UnstructuredMesh(state["idx"], state["xyz"], case["p"], device=DEVICE,
                                    shape=state["shape"])
        bvh = mesh.get_bvh()
        if case["lists"] == "tree":
            return _mesh_outputs(mesh, bvh)
        bvh.build_leaf_maps(mesh).build_grid(0.75)
        out = _mesh_outputs(mesh, bvh)
        out.update(maps=bvh.leaf_maps, start=bvh.grid_start, entries=bvh.grid_entries,
                   boxes=_bits(bvh.grid_boxes))
        return out
    if kind == "boundary":
        b = render.MeshBoundary()
        faces, field = b.execute(state["mesh"], state["fields"]["wave"])
        out = _mesh_outputs(faces, faces.get_bvh())
        out.update(idx=faces.dof_data.ctrl_idx, field_idx=field.ctrl_idx, field=field.packed,
                   elid_faceid=b.elid_faceid)
        return out
    if kind == "surface":
        fb, hits = state["surface"].render(state["camera"], use_lighting=case["lit"])
        return {"colors": fb.colors, "depths": fb.depths, "face": _bits(hits)[:, 0],
                "hit": hits[:, 1:]}
    if kind == "volume":
        fb = state["volume"].render(state["camera"])
        return {"colors": fb.colors, "depths": fb.depths}
    model = state["model"]
    X = model.features(state["mesh"], state["elem"], state["pts"], case["batch"])
    grad, loss = model.grad(X, state["label"], case["batch"], state["weight"], state["ws"])
    model.adam(grad, lr=1e-3)
    return {"grad": grad, "loss": loss, "params": model.params, "m": model.m, "v": model.v}


# ------------------------------------------------------------------- work --

def _sizes(case):
    n, p = case["n"], case["p"]
    hexes = case.get("cells", "hex") == "hex"
    elems = n ** 3 * (1 if hexes else 6)
    nd = (p + 1) ** 3 if hexes else meshgen.tet_dofs(p)
    return elems, nd, (p * n + 1) ** 3


def _step_flops(p, nd):
    """One Newton step: the element's position and three derivatives by sum
    factorisation, and the 3x3 solve."""
    return 2.0 * 3 * (2 * nd + 6 * (p + 1) ** 2 + 9 * (p + 1)) + 120.0


def work(case):
    kind, p = case["kind"], case["p"]
    elems, nd, ctrl = _sizes(case)
    mesh_in = 4 * elems * nd + 12 * ctrl
    if kind == "probe":
        q = case["points"]
        return {"bytes": q * (12 + 8) + min(elems, q) * (nd * 20),
                "flops": q * (3 * _step_flops(p, nd) + 8 * nd)}
    if kind in ("locate", "learned"):
        q = case["points"]
        net = 2 * (128 * (3 * nd + 3) + 128 * 128 + 3 * 128) if kind == "learned" else 0
        return {"bytes": q * (12 + 16) + min(elems, q) * nd * 12,
                "flops": q * (2 * _step_flops(p, nd) + net)}
    if kind == "setup":
        leaves = 33 * elems
        ref = 24 if case["cells"] == "hex" else 48
        out = elems * (12 * nd + 12) + leaves * (64 + 4 + 4 + ref + 43)
        if case["lists"] == "grid":
            out += leaves * (64 + 32) + 12 * leaves * 4
        return {"bytes": mesh_in + out, "flops": leaves * 3 * nd * p * 3.0}
    if kind == "boundary":
        tri = case["cells"] != "hex"
        faces = 6 * case["n"] ** 2 * (2 if tri else 1)
        nd2 = (p + 1) * (p + 2) // 2 if tri else (p + 1) ** 2
        leaves = 17 * faces
        return {"bytes": elems * (4 if tri else 8) * 4 + faces * nd2 * (4 + 4 + 16 + 16) +
                leaves * (64 + 4 + 4 + 24 + 43), "flops": leaves * 3.0 * nd2 * p}
    if kind == "surface":
        rays = case["width"] ** 2
        return {"bytes": rays * (16 + 4 + 20), "flops": rays * 0.4 * 3 * _step_flops(p, (p + 1) ** 2)}
    if kind == "volume":
        rays = case["width"] ** 2
        samples = 0.35 * 0.5 * rays * case["samples"]
        return {"bytes": rays * 20 + elems * nd * 20,
                "flops": samples * (2 * _step_flops(p, nd) + 8 * nd + 150)}
    b, n_in = case["batch"], 3 * (p + 1) ** 3 + 3
    params = 128 * (n_in + 128 + 3) + 259
    return {"bytes": b * (4 + 12 + 12 + 4) + min(b, elems) * nd * 12 + params * 4 * 7,
            "flops": b * 2.0 * (128 * n_in * 2 + 128 * 128 * 3 + 3 * 128 * 3)}


def tolerance(case):
    kind = case["kind"]
    if kind == "probe":
        # Newton tolerance 1e-4 in reference space, quadratic convergence
        return {"rel": 2e-5, "max": 2e-3}
    if kind in ("locate", "learned"):
        # a point within the Newton tolerance of a shared face may go to
        # either element, and its reference point then differs by one
        return {"rel": 5e-3, "max": 0.99, "differ": 1e-4}
    if kind in ("setup", "boundary"):
        # bit-exact trees; the leaf maps are 32-bit inverses
        return {"rel": 1e-6, "max": 1e-4} if case.get("lists") == "grid" else "exact"
    if kind == "surface":
        return {"rel": 2e-3, "max": 0.5, "differ": 2e-3}
    if kind == "volume":
        # a sample on a shared face may be shaded from either element
        return {"rel": 2e-3, "max": 0.5}
    # bf16 operands, gradients summed in any order (Adam's first update has
    # the gradient's sign, so weights with a vanishing gradient may differ)
    return {"rel": 1e-2, "max": 0.99}


# ------------------------------------------------- 64-bit restatements --

def _bernstein(t, p):
    """Basis and derivative [m, p + 1] of the Bernstein polynomials at t."""
    B = torch.stack([math.comb(p, i) * t ** i * (1 - t) ** (p - i) for i in range(p + 1)], -1)
    if p == 1:
        low = torch.ones_like(t)[:, None]
    else:
        low = torch.stack([math.comb(p - 1, i) * t ** i * (1 - t) ** (p - 1 - i)
                           for i in range(p)], -1)
    z = torch.zeros_like(low[:, :1])
    return B, p * (torch.cat([z, low], -1) - torch.cat([low, z], -1))


def _hex_eval(cps, r, p):
    """Values [m, c] and derivatives [m, c, 3] of hex elements with control
    values cps [m, nd, c] (u fastest) at reference points r."""
    m, c = cps.shape[0], cps.shape[2]
    q = cps.view(m, p + 1, p + 1, p + 1, c)
    (Bu, Du), (Bv, Dv), (Bw, Dw) = (_bernstein(r[:, k], p) for k in range(3))

    def dot(u, v, w):
        t = torch.einsum("mkjic,mi->mkjc", q, u)
        t = torch.einsum("mkjc,mj->mkc", t, v)
        return torch.einsum("mkc,mk->mc", t, w)

    return dot(Bu, Bv, Bw), torch.stack([dot(Du, Bv, Bw), dot(Bu, Dv, Bw), dot(Bu, Bv, Dw)], -1)


def _solve(xyz64, idx, n, p, c, pt):
    """Newton for the points pt in the lattice cells c: elements, reference
    points, and whether the solution lies inside."""
    e = (c[:, 2] * n + c[:, 1]) * n + c[:, 0]
    cps = xyz64[idx[e]]
    x = torch.full_like(pt, 0.5)
    for _ in range(12):
        X, J = _hex_eval(cps, x, p)
        dx = torch.linalg.solve_ex(J, (pt - X).unsqueeze(-1))[0].squeeze(-1)
        x = torch.clamp(torch.nan_to_num(x + torch.clamp(dx, -1.0, 1.0), nan=0.5), -0.6, 1.6)
        if float(dx.abs().max()) < 1e-13:
            break
    X, _ = _hex_eval(cps, x, p)
    edge = ((x < 0) & (c == 0)) | ((x > 1) & (c == n - 1))   # flat outer boundary
    inside = ((x >= -1e-9) & (x <= 1 + 1e-9)) | edge
    return e, x, inside.all(1) & ((X - pt).norm(dim=1) < 1e-9)


def _invert(xyz64, idx, n, p, pts):
    """Elements and reference points of pts in a hex lattice mesh over
    [0,1]^3 (-1 outside): Newton in the lattice cell of the point, then step
    by step over the faces that the solution lies beyond, and for the few
    points that this walk does not place, in all the cells around."""
    first = torch.clamp((pts * n).floor().long(), 0, n - 1)
    cell = first.clone()
    el = torch.full((pts.shape[0],), -1, dtype=torch.long, device=DEVICE)
    ref = torch.full_like(pts, -1.0)
    within = ((pts >= 0) & (pts <= 1)).all(1)
    todo = torch.nonzero(within)[:, 0]
    for _ in range(12):
        if todo.numel() == 0:
            break
        c = cell[todo]
        e, x, inside = _solve(xyz64, idx, n, p, c, pts[todo])
        el[todo[inside]], ref[todo[inside]] = e[inside], x[inside]
        move = (x > 1).long() - (x < 0).long()
        cell[todo] = torch.clamp(c + move, 0, n - 1)
        todo = todo[~inside & (cell[todo] != c).any(1)]
    around = sorted(itertools.product(range(-3, 4), repeat=3), key=lambda o: sum(v * v for v in o))
    for o in around:
        todo = torch.nonzero(within & (el < 0))[:, 0]
        if todo.numel() == 0:
            break
        c = torch.clamp(first[todo] + torch.tensor(o, device=DEVICE), 0, n - 1)
        e, x, inside = _solve(xyz64, idx, n, p, c, pts[todo])
        el[todo[inside]], ref[todo[inside]] = e[inside], x[inside]
    return el, ref


def _invert_all(case, xyz, idx, pts, chunk):
    xyz64, n, p = xyz.double(), case["n"], case["p"]
    idx = idx.view(-1, (p + 1) ** 3).long()
    got = [_invert(xyz64, idx, n, p, pts[i:i + chunk].double())
           for i in range(0, pts.shape[0], chunk)]
    return torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])


def _normalize(v):
    return v / v.norm(dim=-1, keepdim=True)


def _camera_rays64(width):
    """Pixel rays of the benchmark camera and its default light's position."""
    c = meshgen.CAMERA
    pos, look_at, up = (torch.tensor(c[k], dtype=torch.float64) for k in ("pos", "look_at", "up"))
    up = _normalize(up)
    look = look_at - pos
    th = math.tan(0.5 * math.radians(c["fov"]))
    ru = torch.linalg.cross(look, up)
    rv = torch.linalg.cross(ru, look)
    light = pos + 0.1 * look.norm() * _normalize(torch.linalg.cross(_normalize(ru), look))
    dx, dy = _normalize(ru) * (2 * th / width), _normalize(rv) * (2 * th / width)
    s = (2.0 * torch.arange(width, dtype=torch.float64) - width) / 2
    d = _normalize(look) + dx * s[None, :, None] + dy * s[:, None, None]
    return pos.to(DEVICE), _normalize(d).reshape(-1, 3).to(DEVICE), light.to(DEVICE)


def _table64(alphas, samples, opacity):
    t = torch.linspace(0, 1, samples, dtype=torch.float64)
    (p0, *a), (p1, *b) = meshgen.TF_RGB
    rgb = torch.stack([a[k] * (1 - t) + b[k] * t for k in range(3)], -1)
    al = torch.ones_like(t)
    if alphas:
        v = [1 - (1 - x) ** opacity for _, x in alphas]
        al = v[0] * (1 - t) + v[1] * t
    return torch.cat([rgb, al[:, None]], -1).to(DEVICE)


def _lookup(table, f, lo, hi):
    s = (torch.clamp(f, lo, hi) - lo) / (hi - lo)
    return table[(s * (table.shape[0] - 1)).long()]


def _surface64(case, xyz, idx, wave):
    """The boundary is the unit cube with undisplaced control points, so the
    rays meet it in closed form; the faces' numbers are left out."""
    n, p, width = case["n"], case["p"], case["width"]
    pos, d, light = _camera_rays64(width)
    t0, t1 = (0.0 - pos) / d, (1.0 - pos) / d
    near, far = torch.minimum(t0, t1), torch.maximum(t0, t1)
    tn, axis = near.max(1)
    hit = (tn < far.min(1)[0]) & (tn > 0)
    X = torch.clamp(pos + tn[:, None] * d, 0, 1)
    other = torch.tensor([[1, 2], [0, 2], [0, 1]], device=DEVICE)[axis]
    uv = X.gather(1, other) * n
    cell2 = torch.clamp(uv.floor(), 0, n - 1)
    uv = uv - cell2
    side = (X.gather(1, axis[:, None])[:, 0] > 0.5).double()
    c = torch.zeros(d.shape[0], 3, dtype=torch.long, device=DEVICE)
    c.scatter_(1, other, cell2.long())
    c.scatter_(1, axis[:, None], (side * (n - 1)).long()[:, None])
    r = torch.zeros_like(X)
    r.scatter_(1, other, uv)
    r.scatter_(1, axis[:, None], side[:, None])
    e = (c[:, 2] * n + c[:, 1]) * n + c[:, 0]
    f = _hex_eval(wave.double()[idx.view(-1, (p + 1) ** 3)[e].long()][..., None], r, p)[0][:, 0]
    # the range of the boundary's own field, which holds the volume's values
    col = _lookup(_table64(None, 1024, 0.0), f, float(wave.min()), float(wave.max()))
    if case["lit"]:
        nrm = torch.zeros_like(X)
        nrm.scatter_(1, axis[:, None], 1.0)
        nrm = torch.where((d * nrm).sum(1, keepdim=True) >= 0, -nrm, nrm)
        col = _blinn_phong(col, nrm, -d, _normalize(light - X), False)
        col[:, :3] = col[:, :3].clamp(0, 1)
    inf = torch.full_like(tn, math.inf)
    zero = torch.zeros_like(tn)
    h = torch.where(hit[:, None], torch.stack([tn, uv[:, 0], uv[:, 1], zero], -1), 0.0)
    return {"colors": torch.where(hit[:, None], col, 0.0), "depths": torch.where(hit, tn, inf),
            "face": None, "hit": h}


def _blinn_phong(c, nrm, view, ld, flip):
    if flip:
        nrm = torch.where((ld * nrm).sum(1, keepdim=True) < 0, -nrm, nrm)
    diffuse = (ld * nrm).sum(1, keepdim=True).clamp(0, 1)
    hv = _normalize(view + ld)
    if flip:
        nrm = torch.where((nrm * hv).sum(1, keepdim=True) < 0, -nrm, nrm)
    shine = (nrm * hv).sum(1, keepdim=True).clamp(0, 1) ** 15.0
    rgb = c[:, :3] * (0.4 + 0.75 * diffuse + 0.8 * shine)
    return torch.cat([rgb, c[:, 3:]], 1)


def _volume64(case, xyz, idx, wave):
    """integrate_partials and the Volume::save compositing, ray by ray."""
    n, p, width, samples = case["n"], case["p"], case["width"], case["samples"]
    pos, d, light = _camera_rays64(width)
    half = 0.5 * 1.001
    t0, t1 = (0.5 - half - pos) / d, (0.5 + half - pos) / d
    near = torch.minimum(t0, t1).max(1)[0].clamp(min=0)
    far = torch.maximum(t0, t1).min(1)[0]
    step = math.sqrt(3.0) / samples
    rays = torch.nonzero(far > near)[:, 0]
    d, near, far = d[rays], near[rays], far[rays]
    steps = int(((far - near) / step).max()) + 1
    table = _table64(meshgen.TF_ALPHA, 1024, 10.0 / samples)
    lo, hi = float(wave.min()), float(wave.max())
    m = rays.numel()
    zero4 = torch.zeros(m, 4, dtype=torch.float64, device=DEVICE)
    color, pixel = zero4.clone(), zero4.clone()
    first = torch.full((m,), math.inf, dtype=torch.float64, device=DEVICE)
    depth = torch.zeros_like(first)
    segment = torch.zeros(m, dtype=torch.long, device=DEVICE)
    in_seg = torch.zeros(m, dtype=torch.bool, device=DEVICE)
    done = near + step >= far
    per = max(1, 400000 // m)
    xyz64, w64, idx = xyz.double(), wave.double(), idx.view(-1, (p + 1) ** 3).long()
    for k0 in range(0, steps, per):
        ks = range(k0, min(k0 + per, steps))
        dist = torch.stack([near + (k + 1) * step for k in ks])
        P = pos + dist[..., None] * d
        use = (dist < far) & ~done
        el = torch.full(dist.shape, -1, dtype=torch.long, device=DEVICE)
        shade = torch.zeros(*dist.shape, 4, dtype=torch.float64, device=DEVICE)
        e, r = _invert(xyz64, idx, n, p, P[use])
        el[use] = e
        ok = e >= 0
        e, r, pt = e[ok], r[ok], P[use][ok]
        f, g = _hex_eval(w64[idx[e]][..., None], r, p)
        c = _lookup(table, f[:, 0], lo, hi)
        if case["lit"]:
            _, J = _hex_eval(xyz64[idx[e]], r, p)
            grad = _normalize(torch.linalg.solve(J.transpose(1, 2), g[:, 0, :, None])[..., 0])
            ld = _normalize(light - pt)
            view = -d.expand(dist.shape[0], -1, -1)[use][ok]
            lit = _blinn_phong(c, grad, view, ld, True)
            lit[:, :3] = lit[:, :3].clamp(0, 1)
            c = torch.where(c[:, 3:] > 0.01, lit, 0.0)
        got = torch.zeros(ok.shape[0], 4, dtype=torch.float64, device=DEVICE)
        got[ok] = c
        shade[use] = got
        for j in range(len(ks)):
            live = ~done
            at = dist[j]
            found = live & (el[j] >= 0)
            begin = found & ~in_seg
            depth = torch.where(begin, at, depth)
            color = torch.where(begin[:, None], 0.0, color)
            a = shade[j][:, 3:] * (1 - color[:, 3:])
            blended = torch.cat([color[:, :3] + shade[j][:, :3] * a, a + color[:, 3:]], 1)
            color = torch.where(found[:, None], blended, color)
            in_seg = in_seg | begin
            end_of_ray = ~(at + step < far)
            full = ~(color[:, 3] < 0.95)
            close = (found & (end_of_ray | full)) | (live & ~found & in_seg)
            head = close & (segment == 0)
            behind = pixel + color * (1 - pixel[:, 3:])
            pixel = torch.where(head[:, None], color, torch.where(close[:, None], behind, pixel))
            first = torch.where(head, depth, first)
            segment = segment + close
            in_seg = in_seg & ~close
            done = done | (live & end_of_ray) | (close & (segment == 5)) | \
                (close & found & (color[:, 3] > 0.95))
    colors = torch.zeros(width * width, 4, dtype=torch.float64, device=DEVICE)
    depths = torch.full((width * width,), math.inf, dtype=torch.float64, device=DEVICE)
    colors[rays], depths[rays] = pixel, first
    return {"colors": colors, "depths": depths}


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _train64(case, gen):
    p = case["p"]
    xyz, idx, elem, pts, label, weight = _pairs(case, gen)
    w = _identity_network(p, gen).double().requires_grad_()
    lay = learned.Layout(p)
    cps = xyz.double()[idx.view(-1, (p + 1) ** 3)[elem.long()].long()]
    lo, hi = cps.min(1)[0], cps.max(1)[0]
    c, h = 0.5 * (lo + hi), 0.5 * (hi - lo).max(1)[0]
    X = (torch.cat([cps, pts.double()[:, None]], 1) - c[:, None]) / h[:, None, None]
    H = _gelu(X.flatten(1) @ w[lay.W1:lay.B1].view(-1, lay.n_in).T + w[lay.B1:lay.W2])
    H = _gelu(H @ w[lay.W2:lay.B2].view(128, 128).T + w[lay.B2:lay.W3])
    Y = H @ w[lay.W3:lay.B3].view(3, 128).T + w[lay.B3:]
    loss = (weight.double()[:, None] * (Y - label.double()) ** 2).sum() / case["batch"]
    loss.backward()
    g = w.grad
    m, v = 0.1 * g, 0.001 * g * g
    new = w.detach() - 1e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return {"grad": g, "loss": loss.detach().reshape(1), "params": new, "m": m, "v": v}


def exact(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "train":
        return _train64(case, gen)
    n, p, cells = case["n"], case["p"], case.get("cells", "hex")
    xyz, idx = _scene(case, seed, gen)
    if kind == "setup":
        # the trees are defined by 32-bit steps; the packed rows have values
        elems, nd, _ = _sizes(case)
        cps = xyz.double()[idx.view(elems, nd).long()]
        rows = (cps - cps[:, :1]).flatten(1)
        pad = -(-(3 * nd + 3) // 4) * 4 - 3 * nd - 3
        packed = torch.cat([rows, cps[:, 0], torch.zeros(elems, pad, device=DEVICE,
                                                         dtype=torch.float64)], 1)
        return {"packed": packed}
    if kind == "boundary" or cells != "hex":
        # integers and 32-bit trees; a tet search without a tree is too slow
        return None
    if kind == "surface":
        return _surface64(case, xyz, idx, _fields(xyz, seed)[0])
    if kind == "volume":
        if case["width"] ** 2 * case["samples"] > 4e7:
            return None   # minutes in 64-bit array operations
        return _volume64(case, xyz, idx, _fields(xyz, seed)[0])
    chunk = 1 << 20 if p < 3 else 1 << 18
    el, ref = _invert_all(case, xyz, idx, _queries(case["points"], gen), chunk)
    if kind != "probe":
        return {"cell": None, "ref": ref}
    out = {}
    conn = idx.view(-1, (p + 1) ** 3)[el.clamp(min=0)].long()
    for k, v in zip(("wave", "blob"), _fields(xyz, seed)):
        f = _hex_eval(v.double()[conn][..., None], ref, p)[0][:, 0]
        out[k] = torch.where(el >= 0, f, -2.0)
    return out
