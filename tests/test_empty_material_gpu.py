"""A material without components, the last 8 bytes of its buffer: it renders
black, and nothing past its MaterialInfo is read (the ordering of paths by
what they hit looks at a material's first component only where there is one).
Every renderer gives the megakernel's image and states."""
import pytest
import torch

from clear_gb300 import _lib
from clear_gb300 import scene as S
from clear_gb300.render import DeviceScene

pytestmark = pytest.mark.gpu

BLOCK = 512  # bytes of a whole block of torch's allocator


def _scene(cuda) -> DeviceScene:
    sc = S.Scene()
    sc.mc.float3_constant_texture("R", 0.5, 0.5, 0.5)
    sc.mc.float_constant_texture("sigma0", 0.0)
    sc.mc.float3_constant_texture("M", 20.0, 20.0, 20.0)
    sc.mc.matte_material("m", None, "R", "sigma0")
    sc.mc.diffuse_light_property("light", "M")
    sc.begin_object()
    for x, y, z in ((-1.0, -1.0, 0.0), (1.0, -1.0, 0.0), (1.0, 1.0, 0.0), (-1.0, 1.0, 0.0)):
        sc.add_vertex(x, y, z)
    sc.add_face((0, 1, 2), sc.mat_ref["m"])
    sc.add_face((0, 2, 3), sc.mat_ref["m"], light=sc.light_ref["light"])
    sc.end_object()
    sc.set_camera(32, 32, S.look_at((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (0, 1, 0)), fov_y_deg=40.0)
    sc.build()
    ds = DeviceScene(sc, cuda)
    # the materials again with an empty one behind them, up to the end of a block
    blob = ds.t["materials"]
    pad = -blob.numel() % 4
    at = blob.numel() + pad
    size = (at + 8 + BLOCK - 1) // BLOCK * BLOCK
    buf = torch.zeros(size, dtype=torch.uint8, device=cuda)
    first = size - 8 - at
    buf[first:first + blob.numel()] = blob
    ds.t["materials"] = buf
    ds.c.materials = buf.data_ptr() + first
    # both faces' material references (byte 52 of a 56-byte Face)
    faces = ds.t["faces"].view(torch.int16).view(-1, 28)
    assert int(faces[0, 26]) == sc.mat_ref["m"]
    faces[:, 26] = at
    return ds


@pytest.mark.parametrize("ordered", [False, True])
def test_material_without_components(cuda, ordered):
    ds = _scene(cuda)
    want_rng, want = ds.new_frame()
    ds.render(want_rng, want, 4, max_depth=4, ordered=ordered, wavefront=False)
    rng, pix = ds.new_frame()
    ds.render(rng, pix, 4, max_depth=4, ordered=ordered, wavefront=True)
    torch.cuda.synchronize()
    assert torch.equal(pix, want) and torch.equal(rng, want_rng)
    lit = int((pix[:, :3].amax(dim=1) > 0).sum())
    assert 300 < lit < 700  # the lamp's half of the square; the other half, and the lamp's reflection, black
    assert _lib.device_status() == 0
