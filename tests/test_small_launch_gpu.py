"""The launch shapes for few queries and few rays against the ones for many:
the same queries and rays give the same bits."""
import pytest

from devil_ray_b200 import _lib as L
from devil_ray_b200 import api, meshgen, render

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


# rays from one to the largest numbers that 32, 16 and 8 lanes a ray take and
# one more; above half the SMs' lanes (the whole frame) it is one lane
@pytest.mark.parametrize("kind,p,lit", [("hex", 1, True), ("hex", 2, False), ("hex", 3, True),
                                        ("tet", 2, True)])
def test_few_rays_equal_many(cuda, kind, p, lit):
    import torch
    m, shape = _mesh(kind, 4, p)
    mesh = api.UnstructuredMesh(m.ctrl_idx, m.xyz, m.order, device=cuda, shape=shape)
    values = torch.sin(7.0 * torch.as_tensor(m.xyz, device=cuda)).sum(1).float()
    field = render.UnstructuredField(m.ctrl_idx, values, m.order, device=cuda, shape=shape)
    c = meshgen.CAMERA
    camera = render.Camera(512, 512, c["pos"], c["look_at"], c["up"], c["fov"])
    light = [render.PointLight.default(camera)]
    active = render.cull_rays(camera.create_rays(cuda), mesh.bounds())
    lanes = 512 * torch.cuda.get_device_properties(cuda).multi_processor_count
    sizes = [1, 100, 6 * lanes // 32, 6 * lanes // 32 + 1, 6 * lanes // 16, 6 * lanes // 16 + 1,
             lanes // 2]
    assert active.shape[0] > max(lanes // 2, sum(sizes))
    # at the larger opacities rays end within a few samples, some of them
    # before their group would take them over
    for opacity in (0.02, 0.9, 0.9999, 1.0):
        vol = render.Volume(mesh, field)
        table = render.ColorTable()
        table.add_point(0.0, (0.1, 0.2, 0.9))
        table.add_point(1.0, (0.9, 0.4, 0.1))
        table.add_alpha(0.0, 0.0)
        table.add_alpha(1.0, opacity)
        vol.color_map().color_table(table)
        vol.samples(37)
        vol.use_lighting(lit)
        whole, stats = vol.render(camera, light, active=active, stats=True)
        colors, depths = whole.colors.clone(), whole.depths.clone()
        parts = torch.zeros_like(colors)
        first, got = 0, []
        fb = render.Framebuffer(512, 512, cuda)
        seen = torch.full_like(depths, float("inf"))
        for size in sizes:
            some = active[first:first + size].contiguous()
            _, st = vol.render(camera, light, fb=fb, active=some, stats=True)
            hit = torch.isfinite(fb.depths)
            parts[hit], seen[hit] = fb.colors[hit], fb.depths[hit]
            got.append([s[:some.shape[0]].clone() for s in st])
            first += some.shape[0]
        for k in range(3):
            assert torch.equal(torch.cat([g[k] for g in got]), stats[k][:first])
        done = torch.isfinite(seen)
        assert done.sum() > 1000
        assert torch.equal(parts[done], colors[done]) and torch.equal(seen[done], depths[done])


# the partials of a few rays, in both parts of their march, against the same
# rays among many
@pytest.mark.parametrize("opacity", [0.02, 0.9, 1.0])
def test_partials_of_few_rays_equal_many(cuda, opacity):
    import torch
    m, shape = _mesh("hex", 4, 2)
    mesh = api.UnstructuredMesh(m.ctrl_idx, m.xyz, m.order, device=cuda, shape=shape)
    values = torch.sin(9.0 * torch.as_tensor(m.xyz, device=cuda)).sum(1).float()
    field = render.UnstructuredField(m.ctrl_idx, values, m.order, device=cuda, shape=shape)
    c = meshgen.CAMERA
    camera = render.Camera(512, 512, c["pos"], c["look_at"], c["up"], c["fov"])
    vol = render.Volume(mesh, field)
    table = render.ColorTable()
    table.add_point(0.0, (0.1, 0.2, 0.9))
    table.add_point(1.0, (0.9, 0.4, 0.1))
    table.add_alpha(0.0, 0.0)
    table.add_alpha(1.0, opacity)
    vol.color_map().color_table(table)
    vol.samples(60)
    light = [render.PointLight.default(camera)]
    rays = camera.create_rays(cuda)
    some = rays[torch.arange(0, rays.shape[0], 37, device=cuda)].contiguous()
    many, few = vol.integrate(rays, light), vol.integrate(some, light)
    pixel = many[:, 0].contiguous().view(torch.int32)
    kept = many[(pixel % 37 == 0).nonzero().squeeze(1)]
    assert few.shape[0] > 500
    assert torch.equal(few.view(torch.int32), kept.view(torch.int32))


# a configuration that is given decides the launch at every size: with the
# order there are launches before the locate kernel, with staged results one
# behind it, without order or configuration there is one in all
@pytest.mark.parametrize("entry", ["batched", "noalloc"])
def test_a_given_configuration_holds_for_few_queries(cuda, entry):
    import ctypes as C
    import torch
    m, shape = _mesh("hex", 5, 2)
    g = api.UnstructuredMesh(m.ctrl_idx, m.xyz, m.order, device=cuda, shape=shape)
    q = torch.as_tensor(meshgen.uniform_queries(5000, 3), device=cuda)
    bd = g.get_bvh().desc()
    md = g.desc()
    opts = L.DrbNewtonOpts(1e-5, 20, L.GUESS_ELEM_CENTER, None)
    fn = L.lib().drb_locate_batched if entry == "batched" else L.lib().drb_locate_batched_noalloc
    out = []

    def launches(cfg):
        cell = torch.empty(5000, dtype=torch.int32, device=cuda)
        ref = torch.empty((5000, 3), dtype=torch.float32, device=cuda)
        first = L.lib().drb_kernel_launches()
        assert fn(C.byref(md), C.byref(bd), C.c_void_p(q.data_ptr()), 5000, C.byref(opts),
                  None if cfg is None else C.byref(cfg), C.c_void_p(cell.data_ptr()),
                  C.c_void_p(ref.data_ptr()), L.DrbQueryStats(),
                  C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        out.append((cell, ref))
        return L.lib().drb_kernel_launches() - first

    assert launches(None) == 1
    ordered = launches(L.DrbLocateConfig(128, 0, 64, 1, 0))
    assert ordered > 1
    if entry == "batched":
        staged = launches(L.DrbLocateConfig(128, 0, 64, 2, 0))
        assert launches(L.DrbLocateConfig(128, 0, 64, 3, 0)) == staged + 1
    assert launches(L.DrbLocateConfig(128, 1, 64, 0, 1)) == 1
    for cell, ref in out[1:]:
        assert torch.equal(cell, out[0][0])
        assert torch.equal(ref.view(torch.int32), out[0][1].view(torch.int32))
