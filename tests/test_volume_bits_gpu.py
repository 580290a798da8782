"""Lit volume frames against stored ones, bit for bit.

The stored frames were written by the renderer whose shading divides: the
gradient times the explicit inverse (matrix_inverse, matrix.hpp:430-456) and
each normalisation one division a component.  A cheaper form that rounds
differently shows here in the last bits, and in the coherent marches, which
start a sample from the previous one's factors, also as samples on shared
faces that fall to the other element.

    python tests/test_volume_bits_gpu.py writes the file."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "volume_frames.npz"
WIDTH = 28
# mesh kind, elements an axis, order, march (0 plain, 1 linear, 2 quadratic
# predictor)
FRAMES = {"hex_p1_coherent": ("hex", 6, 1, 1), "hex_p2_plain": ("hex", 6, 2, 0),
          "hex_p3_coherent": ("hex", 5, 3, 1), "hex_p3_quadratic": ("hex", 5, 3, 2),
          "tet_p2_coherent": ("tet", 4, 2, 1)}


def frame(name, device):
    """Colours [WIDTH^2, 4] of one lit frame."""
    import torch
    from devil_ray_b200 import _lib as L
    from devil_ray_b200 import api, meshgen, render
    kind, n, p, march = FRAMES[name]
    if kind == "tet":
        m, shape = meshgen.tet_warped_mesh(n, p, 0.05, jitter=0.01, seed=5), L.SHAPE_SIMPLEX
    else:
        m, shape = meshgen.warped_mesh(n, p, 0.08, jitter=0.01, seed=5), L.SHAPE_TENSOR
    mesh = api.UnstructuredMesh(m.ctrl_idx, m.xyz, m.order, device=device, shape=shape)
    x = m.xyz.astype(np.float64)
    values = (x[:, 0] * x[:, 1] + x[:, 2] ** 2 - 0.7 * x[:, 0]).astype(np.float32)
    field = render.UnstructuredField(m.ctrl_idx, values, m.order, device=device, shape=shape)
    c = meshgen.CAMERA
    camera = render.Camera(WIDTH, WIDTH, c["pos"], c["look_at"], c["up"], c["fov"])
    vol = render.Volume(mesh, field)
    table = render.ColorTable()
    table.add_point(0.0, (0.1, 0.2, 0.9))
    table.add_point(1.0, (0.9, 0.4, 0.1))
    table.add_alpha(0.0, 0.05)
    table.add_alpha(1.0, 0.3)
    vol.color_map().color_table(table)
    vol.samples(60)
    vol.use_lighting(True)
    vol.coherent = march
    fb = vol.render(camera, [render.PointLight.default(camera)])
    torch.cuda.synchronize()
    return fb.colors.cpu().numpy().reshape(-1, 4)


@pytest.mark.parametrize("name", list(FRAMES))
def test_lit_frame_keeps_its_bits(cuda, name):
    want = np.load(GOLDEN)[name]
    got = frame(name, cuda)
    assert (want[:, 3] > 0.3).mean() > 0.3
    assert np.array_equal(got.view(np.int32), want.view(np.int32))


if __name__ == "__main__":
    np.savez_compressed(GOLDEN, **{name: frame(name, "cuda") for name in FRAMES})
