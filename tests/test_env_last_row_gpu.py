"""The density of paths that leave straight down: the environment's last row.

acosf(-1) / pi is exactly 1 in float32, the end of the importance distribution.
Such a path reads the first row's texel (the image lookup wraps) and the last
row's density, which enters through the weight of multiple importance sampling.
The rows' densities differ by four orders of magnitude here, so the weight on
the adjoint's tape tells the rows apart; it is evaluated again in 64 bits from
the scene's blob.  The renderers share that lookup: the same image from all."""
import numpy as np
import pytest
import torch

from clear_gb300 import _lib
from clear_gb300 import scene as S
from clear_gb300.batch import BatchRenderer
from clear_gb300.render import TAPE_WORDS, DeviceScene

pytestmark = pytest.mark.gpu

SIZE, SPP, ROWS, COLS = 48, 64, 8, 16
EMIT, SAMPLE = 1, 4


def _scene() -> S.Scene:
    sc = S.Scene()
    mc = sc.mc
    mc.float3_constant_texture("Rs", 0.9, 0.9, 0.9)
    mc.float3_constant_texture("Rd", 0.0, 0.0, 0.0)
    mc.float_constant_texture("n", 1.0e5)
    mc.ashikhmin_material("glossy", None, "Rs", "Rd", "n", "n")
    sc.begin_object()
    for x, z in ((-1.0, -1.0), (1.0, -1.0), (1.0, 1.0), (-1.0, 1.0)):
        sc.add_vertex(x, 1.0, z)
    sc.add_face((0, 1, 2), sc.mat_ref["glossy"])
    sc.add_face((0, 2, 3), sc.mat_ref["glossy"])
    sc.end_object()
    rgba = np.ones((ROWS, COLS, 4), dtype=np.float16)
    rgba[..., :3] = (10.0 ** np.linspace(2.0, -2.0, ROWS))[:, None, None].astype(np.float16)
    mc.image_texture("env", rgba, "rgba16f")
    mc.image_based_env_light_property("IBL", "env", rgba[..., :3].astype(np.float32), 1.0)
    sc.set_environment("IBL")
    sc.set_camera(SIZE, SIZE, S.look_at((0.0, -1.0, 0.0), (0.0, 1.0, 0.0), (0, 0, 1)), fov_y_deg=0.5)
    sc.build()
    return sc


def _row_densities(ds: DeviceScene) -> np.ndarray:
    """pdf over (u, v) in every row (rows of one value: 1 along u)."""
    blob = np.ascontiguousarray(ds.blobs["others"]).view(np.uint8).reshape(-1)
    head = ds.env_dist["dist_offset"] + 8  # the distribution over rows
    num, off_pdf = int(blob[head + 4:head + 8].view(np.uint32)[0]), int(blob[head + 20:head + 24].view(np.int32)[0])
    assert num == ROWS
    return blob[head + off_pdf:head + off_pdf + 4 * ROWS].view(np.float32).astype(np.float64)


def test_weight_comes_from_the_last_row(cuda):
    sc = _scene()
    ds = DeviceScene(sc, cuda)
    pdf = _row_densities(ds)
    assert pdf[0] / pdf[-1] > 5e3
    rng, pix = ds.new_frame()
    dloss = torch.ones_like(pix)
    none = torch.zeros(0, dtype=torch.int32, device=cuda)
    grad_env = torch.zeros((ROWS * COLS, 4), dtype=torch.float32, device=cuda)
    tape = torch.zeros((8 * SIZE * SIZE * SPP, TAPE_WORDS), dtype=torch.int32, device=cuda)
    count = torch.zeros(1, dtype=torch.int32, device=cuda)
    ds.render_adjoint(rng, dloss, SPP, 2, none, none.to(torch.uint8), torch.zeros((0, 4), device=cuda),
                      sc.tex_ref["env"], grad_env, tape, count)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0 and int(count.item()) <= tape.shape[0]
    rec = tape[:int(count.item())].cpu().numpy()
    f = rec.view(np.float32).astype(np.float64)
    kind = rec[:, 3] & 0xFF
    down = (kind == EMIT) & (rec[:, 2] == 1) & (rec[:, 8] >= 0) & (rec[:, 8] < COLS)
    assert down.sum() >= 20
    cos_by_pdf = {tuple(r): c for r, c in zip(rec[(kind == SAMPLE) & (rec[:, 2] == 0), :2].tolist(),
                                              zip(f[(kind == SAMPLE) & (rec[:, 2] == 0), 4],
                                                  f[(kind == SAMPLE) & (rec[:, 2] == 0), 18]))}
    # 2 pi^2 sin(theta) at theta = float32(pi); |.|: only its square counts
    area = abs(2.0 * np.float64(np.float32(np.pi)) ** 2 * np.sin(np.float64(np.float32(np.pi))))
    for r, w in zip(rec[down, :2].tolist(), f[down, 4]):
        ratio, cos = cos_by_pdf[tuple(r)]
        p_bsdf = abs(cos) / ratio
        p_light = pdf[-1] / area
        want = p_bsdf ** 2 / (p_light ** 2 + p_bsdf ** 2)
        assert 1e-6 < want < 1.0 - 1e-6
        # a handful of float32 roundings and the 2 ulp of sinf, squared: below 1e-5
        assert abs(w - want) <= 1e-5 * want, (w, want)


def test_renderers_agree(cuda):
    sc = _scene()
    ds = DeviceScene(sc, cuda)
    frames = []
    for wavefront in (False, True):
        rng, pix = ds.new_frame()
        ds.render(rng, pix, SPP, max_depth=2, wavefront=wavefront)
        frames.append((pix, rng))
    br = BatchRenderer([sc], cuda)
    rng, pix = br.new_frame()
    br.render(rng, pix, SPP, 2)
    frames.append((pix, rng))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    for pix, rng in frames[1:]:
        assert torch.equal(pix, frames[0][0]) and torch.equal(rng, frames[0][1])
