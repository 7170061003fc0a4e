"""The megakernel's searches test boxes by Woo's test alone where they follow the
reference's order (also every scene with cutouts), the wavefront's classify them
first: the same images and random states, bit for bit, in both orders."""
import numpy as np
import pytest
import torch

from clear_gb300 import _lib, scenes
from clear_gb300 import scene as S
from clear_gb300.batch import random_scene
from clear_gb300.render import SCENE_ALPHA, DeviceScene, scene_flags

pytestmark = pytest.mark.gpu


def _with_cutouts(make, monkeypatch) -> S.Scene:
    """The scene with a square of checkered alpha in front of it."""
    build = S.Scene.build

    def build_with(sc):
        rgba = np.zeros((4, 4, 4), dtype=np.uint8)
        rgba[..., 3] = 255 * ((np.arange(4)[:, None] + np.arange(4)[None, :]) % 2)
        sc.mc.image_texture("cut", rgba, "rgba8")
        mat = next(iter(sc.mat_ref.values()))
        sc.begin_object()
        for x, y in ((0.2, 0.2), (0.8, 0.2), (0.8, 0.8), (0.2, 0.8)):
            sc.add_vertex(x, y, 0.9)
        for uv in ((0.0, 0.0), (1.0, 0.0), (1.0, 1.0), (0.0, 1.0)):
            sc.add_uv(*uv)
        for tri in ((0, 1, 2), (0, 2, 3)):
            sc.add_face(tri, mat, uv=tri, alpha_tex=sc.tex_ref["cut"])
        sc.end_object()
        build(sc)

    with monkeypatch.context() as m:
        m.setattr(S.Scene, "build", build_with)
        return make()


@pytest.mark.parametrize("cutouts", [False, True])
@pytest.mark.parametrize("kind", ["cornell", "random"])
def test_megakernel_equals_wavefront(cuda, monkeypatch, kind, cutouts):
    make = {"cornell": lambda: scenes.cornell_box(48, 40), "random": lambda: random_scene(3000, 48, 40, 5)}[kind]
    sc = _with_cutouts(make, monkeypatch) if cutouts else make()
    assert (scene_flags(sc.blobs()) == SCENE_ALPHA) == cutouts
    ds = DeviceScene(sc, cuda)
    images = []
    for ordered in (False, True):
        for wavefront in (False, True):
            rng, pix = ds.new_frame()
            ds.render(rng, pix, 4, max_depth=6, ordered=ordered, wavefront=wavefront)
            images.append((pix, rng))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0 and float(images[0][0].max()) > 0
    for pix, rng in images[1:]:
        assert torch.equal(pix, images[0][0]) and torch.equal(rng, images[0][1])
