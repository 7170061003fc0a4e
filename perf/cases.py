"""The work this framework is used for, as measurable cases.

Each case is one call (or one frame, or one gradient step) through the
package's public interface.  Four families: ``build`` (one LBVH per
call), ``build_batched`` (many scenes per call), ``trace`` (ray queries
against a built tree) and ``render`` (whole frames, gradient steps and
batches of scenes).  ``listed()`` names the fixed cases, ``draw(rng)`` takes
one more from the same ranges; ``prepare`` makes what a program holds before
the call, ``run`` makes the call, ``work`` states the bytes and operations no
implementation can avoid, ``exact`` gives the 64-bit answer where one can be
computed directly.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from clear_gb300 import _lib, batch, lbvh, postprocess, scenes
from clear_gb300.render import DeviceScene

MI = 1 << 20


def listed() -> list[dict]:
    return [
        # The size and key width of the reference's own published build
        # figure: a model of about 35,000 triangles, 20 bits per axis.  An
        # interactive viewer rebuilds such a model every frame, so launches
        # and latency count.
        {"name": "build_model", "family": "build", "mesh": "grid", "tris": 34848, "bits": 20},
        # An ordinary scene: a triangle list of no particular size.
        {"name": "build_scene", "family": "build", "mesh": "soup", "tris": 1000003, "bits": 10},
        # The largest scene of the build benchmark.
        {"name": "build_large", "family": "build", "mesh": "soup", "tris": 16 * MI, "bits": 10},
        # The batch benchmark's scenes (512, log-uniform in [1 k, 200 k]),
        # rebuilt together in one call.
        {"name": "build_batch", "family": "build_batched", "scenes": 512, "min_tris": 1000, "max_tris": 200000,
         "bits": 10},
        # Picking and range queries: about a thousand rays a call against a
        # model, latency-bound.
        {"name": "trace_pick", "family": "trace", "query": "closest", "order": "nearer", "rays_of": "random",
         "rays": 1000, "mesh": "grid", "tris": 34848},
        # Primary visibility: a full-HD camera's rays over a 2 M-triangle
        # terrain mesh (neighbouring rays go together).
        {"name": "trace_camera", "family": "trace", "query": "closest", "order": "nearer", "rays_of": "camera",
         "width": 1920, "height": 1080, "rays": 1920 * 1080, "mesh": "grid", "tris": 2 * 1024 * 1024},
        # Incoherent ray lists from outside the path tracer, in the form the
        # documentation advises for them (sorted by origin).
        {"name": "trace_scattered", "family": "trace", "query": "closest", "order": "sorted", "rays_of": "random",
         "rays": 8 * MI, "mesh": "soup", "tris": 4 * MI},
        # Visibility between pairs of points in the order they come.
        {"name": "trace_shadow", "family": "trace", "query": "shadow", "order": "given", "rays_of": "segments",
         "rays": 4 * MI, "mesh": "soup", "tris": 4 * MI},
        # The small path-tracing benchmark, to the finished 8-bit image.
        {"name": "render_cornell", "family": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 5},
        # The large path-tracing benchmark (full HD, 2.2 M triangles, thin
        # lens, sky, bump maps), some samples of a progressive render.
        {"name": "render_terrain", "family": "render", "scene": "terrain", "width": 1920, "height": 1080, "spp": 8,
         "depth": 8},
        # A gradient step of inverse rendering: the image, the loss gradient,
        # the gradients of 16 material parameters and the environment texels.
        {"name": "gradient_step", "family": "render", "scene": "gradient", "width": 512, "height": 512, "spp": 8,
         "depth": 5},
        # Many small scenes rendered by one launch.
        {"name": "render_batch", "family": "render", "scene": "batch", "scenes": 64, "min_tris": 1000,
         "max_tris": 200000, "spp": 2, "depth": 5},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["build", "build", "build", "build_batched", "trace", "trace", "trace", "trace", "frame",
                       "gradient", "batch"])
    mesh = rng.choice(["soup", "grid"])
    if kind == "build":
        return {"family": "build", "mesh": mesh, "tris": _log_int(rng, 1000, 16 * MI), "bits": rng.choice([10, 10, 20])}
    if kind == "build_batched":
        return {"family": "build_batched", "scenes": _log_int(rng, 8, 512), "min_tris": 1000,
                "max_tris": _log_int(rng, 5000, 200000), "bits": 10}
    if kind == "trace":
        query = rng.choice(["closest", "closest", "shadow"])
        case = {"family": "trace", "query": query, "mesh": mesh, "tris": _log_int(rng, 1000, 4 * MI)}
        if query == "shadow":
            case.update(order=rng.choice(["given", "sorted"]), rays_of="segments", rays=_log_int(rng, 1000, 4 * MI))
            return case
        case["order"] = rng.choice(["nearer", "nearer", "sorted", "reference"])
        if rng.random() < 0.5:
            w, h = _log_int(rng, 64, 1920), _log_int(rng, 64, 1080)
            case.update(rays_of="camera", width=w, height=h, rays=w * h)
        else:
            case.update(rays_of="random",
                        rays=_log_int(rng, 1000, 1 * MI if case["order"] == "reference" else 8 * MI))
        return case
    if kind == "frame":
        if rng.random() < 0.5:
            return {"family": "render", "scene": "cornell", "width": _log_int(rng, 96, 512),
                    "height": _log_int(rng, 96, 512), "spp": rng.randint(2, 16), "depth": rng.randint(3, 8)}
        return {"family": "render", "scene": "terrain", "width": _log_int(rng, 320, 1920),
                "height": _log_int(rng, 240, 1080), "spp": rng.randint(1, 8), "depth": rng.randint(3, 8)}
    if kind == "gradient":
        return {"family": "render", "scene": "gradient", "width": _log_int(rng, 64, 512),
                "height": _log_int(rng, 64, 512), "spp": rng.randint(2, 8), "depth": rng.randint(3, 5)}
    return {"family": "render", "scene": "batch", "scenes": _log_int(rng, 8, 64), "min_tris": 1000,
            "max_tris": _log_int(rng, 5000, 200000), "spp": rng.randint(1, 2), "depth": rng.randint(3, 5)}


# ---------------------------------------------------------------- geometry


def _generator(seed: int, device) -> torch.Generator:
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _unit(shape, g, device) -> torch.Tensor:
    d = torch.randn(shape, generator=g, device=device)
    return d / d.norm(dim=-1, keepdim=True).clamp_min(1e-20)


def _soup(n: int, seed: int, device):
    """Triangles scattered in the unit cube, edges of about half the mean
    spacing: the distribution of the build benchmark."""
    g = _generator(seed, device)
    c = torch.rand((n, 1, 3), generator=g, device=device)
    edge = torch.empty((n, 3, 1), device=device).exponential_(generator=g) * (0.5 * n ** (-1.0 / 3.0))
    v = (c + _unit((n, 3, 3), g, device) * edge).view(3 * n, 3)
    return tuple(v[:, k].contiguous() for k in range(3)), None, n


def _grid(n: int, seed: int, device):
    """A heightfield mesh of n triangles over the unit square: shared
    vertices, smooth relief, faces row by row."""
    g = _generator(seed, device)
    side = max(2, math.ceil(math.sqrt(n / 2)) + 1)
    u = torch.linspace(0.0, 1.0, side, device=device)
    z, x = torch.meshgrid(u, u, indexing="ij")
    y = torch.zeros_like(x)
    for octave in range(6):
        a = (torch.rand(2, generator=g, device=device) + 0.5) * (6.0 * 2 ** octave)
        p = torch.rand(2, generator=g, device=device) * 6.2831853
        y += 0.15 * 0.5 ** octave * torch.sin(a[0] * x + p[0]) * torch.sin(a[1] * z + p[1])
    i = torch.arange(side - 1, device=device, dtype=torch.int32)
    a = (i[:, None] * side + i[None, :]).reshape(-1)
    faces = torch.stack([torch.stack([a, a + side, a + 1], -1), torch.stack([a + 1, a + side, a + side + 1], -1)], 1)
    return (x.reshape(-1), y.reshape(-1), z.reshape(-1)), faces.reshape(-1, 3)[:n].contiguous(), n


def _mesh(case: dict, seed: int, device):
    return (_grid if case["mesh"] == "grid" else _soup)(case["tris"], seed, device)


def _rays(case: dict, seed: int, device) -> torch.Tensor:
    """8 floats a ray: origin, tmax, direction, 0."""
    g = _generator(seed + 1000003, device)
    m = case["rays"]
    r = torch.zeros((m, 8), device=device)
    if case["rays_of"] == "camera":
        # a camera above the scene's edge looking at its middle; one jittered
        # ray per pixel, pixels in row order
        w, h = case["width"], case["height"]
        eye = torch.tensor([0.5, 0.9, 1.6], device=device) + 0.05 * torch.randn(3, generator=g, device=device)
        fwd = torch.tensor([0.5, 0.1, 0.4], device=device) - eye
        fwd = fwd / fwd.norm()
        right = torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device=device))
        right = right / right.norm()
        up = torch.linalg.cross(right, fwd)
        j = torch.rand((2, m), generator=g, device=device)
        p = torch.arange(m, device=device)
        sx = ((p % w) + j[0] - 0.5 * w) / h
        sy = (0.5 * h - torch.div(p, w, rounding_mode="floor") - j[1]) / h
        d = fwd + (0.75 * sx)[:, None] * right + (0.75 * sy)[:, None] * up
        r[:, 0:3] = eye
        r[:, 3] = math.inf
        r[:, 4:7] = d / d.norm(dim=-1, keepdim=True)
    elif case["rays_of"] == "segments":
        a = torch.rand((m, 3), generator=g, device=device)
        d = torch.rand((m, 3), generator=g, device=device) - a
        length = d.norm(dim=-1).clamp_min(1e-12)
        r[:, 0:3] = a
        r[:, 3] = length
        r[:, 4:7] = d / length[:, None]
    else:
        r[:, 0:3] = torch.rand((m, 3), generator=g, device=device) * 1.2 - 0.1
        r[:, 3] = math.inf
        r[:, 4:7] = _unit((m, 3), g, device)
    return r


def _batch_sizes(case: dict, seed: int):
    """Triangle count, width, height and seed of every scene of a batch: the
    sizes of the batch benchmark, the scenes' contents by `seed`."""
    sizes = batch.batch_workload(case["scenes"], min_tris=case["min_tris"], max_tris=case["max_tris"])
    return [(n, w, h, (s + 611953 * seed) % (1 << 31)) for n, w, h, s in sizes]


def _pixel_states(n: int, seed: int, device) -> torch.Tensor:
    g = _generator(seed + 7000003, device)
    return torch.randint(1, 2 ** 31 - 1, (n, 4), generator=g, device=device, dtype=torch.int32)


# ------------------------------------------------------------ prepare, run


def prepare(case: dict, seed: int) -> dict:
    device = torch.device("cuda")
    family = case["family"]
    state = {"case": case}
    if family == "build":
        state["vertices"], state["faces"], n = _mesh(case, seed, device)
        state["builder"] = lbvh.LBVHBuilder(n, device)
    elif family == "build_batched":
        sizes = [s[0] for s in _batch_sizes(case, seed)]
        state["offsets"] = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64).tolist()
        n = state["offsets"][-1]
        # every scene a soup of its own density in the unit cube
        g = _generator(seed, device)
        per = torch.tensor(sizes, device=device, dtype=torch.float32).pow(-1.0 / 3.0)
        per = per.repeat_interleave(torch.tensor(sizes, device=device))
        edge = torch.empty((n, 3, 1), device=device).exponential_(generator=g) * (0.5 * per)[:, None, None]
        v = (torch.rand((n, 1, 3), generator=g, device=device) + _unit((n, 3, 3), g, device) * edge).view(3 * n, 3)
        state["vertices"] = tuple(v[:, k].contiguous() for k in range(3))
        state["builder"] = lbvh.LBVHBuilder(n, device)
        # the buffers the scenes are rendered from, rebuilt in place (a scene
        # of n triangles writes n - 1 of its n node slots)
        state["bvh"] = lbvh.BatchBVH(state["offsets"], case["bits"], device)
        state["bvh"].nodes.zero_()
        state["offsets_c"] = (C.c_uint32 * len(sizes + [0]))(*state["offsets"])
    elif family == "trace":
        vertices, faces, n = _mesh(case, seed, device)
        state["bvh"] = lbvh.LBVHBuilder(n, device).perform(vertices, faces, n, 10)
        state["rays"] = _rays(case, seed, device)
        torch.cuda.synchronize()  # the builder and its scratch go with this scope
    elif case["scene"] == "batch":
        made = [batch.random_scene(*s) for s in _batch_sizes(case, seed)]
        state["renderer"] = batch.BatchRenderer(made, device)
        state["states"] = _pixel_states(state["renderer"].total_pixels, seed, device)
    elif case["scene"] == "gradient":
        r = np.random.default_rng(seed)
        albedo = [np.clip(np.asarray(m[2]) + r.normal(0.0, 0.05, 3), 0.05, 0.95) for m in scenes.ADJ_MATERIALS]
        sc, info = scenes.cornell_adjoint(case["width"], case["height"], albedo=albedo)
        ds = state["scene"] = DeviceScene(sc, device)
        tex = info["albedo_tex"] + info["rough_tex"]
        state["tex"] = torch.tensor(tex, dtype=torch.int32, device=device)
        state["kind"] = torch.tensor([0] * 8 + [1] * 8, dtype=torch.uint8, device=device)
        state["env_tex"], (eh, ew) = info["env_tex"], info["env_shape"]
        state["env_texels"] = eh * ew
        n = ds.width * ds.height
        state["target"] = 0.05 * torch.rand((n, 4), generator=_generator(seed, device), device=device)
        state["states"] = _pixel_states(n, seed, device)
    else:
        r = np.random.default_rng(seed)
        if case["scene"] == "cornell":
            albedos = {k: tuple(map(float, r.uniform(0.05, 0.85, 3))) for k in ("red", "green", "white", "base")}
            sc = scenes.cornell_box(case["width"], case["height"], albedos=albedos)
        else:
            # the benchmark's own terrain; the seed chooses the paths
            sc = scenes.terrain_scene(case["width"], case["height"])
        ds = state["scene"] = DeviceScene(sc, device)
        state["states"] = _pixel_states(ds.width * ds.height, seed, device)
    return state


def run(state: dict):
    case = state["case"]
    family = case["family"]
    if family == "build":
        bvh = state["builder"].perform(state["vertices"], state["faces"], case["tris"], case["bits"])
        # word 3 of the root record is a reference, not a number: the record's bits
        return {"nodes": bvh.nodes, "tris": bvh.tris, "root": bvh.root_box.view(torch.int32)}
    if family == "build_batched":
        b, (vx, vy, vz) = state["bvh"], state["vertices"]
        _lib.call("clr_lbvh_build_batched", state["builder"]._h, vx.data_ptr(), vy.data_ptr(), vz.data_ptr(), None,
                  state["offsets_c"], len(b), case["bits"], 8, b.nodes.data_ptr(), b.tris.data_ptr(),
                  b.root_boxes.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"nodes": b.nodes, "tris": b.tris, "roots": b.root_boxes.view(torch.int32)}
    if family == "trace":
        if case["query"] == "shadow":
            return {"occluded": lbvh.trace_shadow(state["bvh"], state["rays"], sort=case["order"] == "sorted")}
        ids, ts = lbvh.trace_closest(state["bvh"], state["rays"], ordered=case["order"] != "reference",
                                     sort=case["order"] == "sorted")
        return {"id": ids, "t": ts}
    spp, depth = case["spp"], case["depth"]
    rng = state["states"].clone()
    if case["scene"] == "batch":
        pix = torch.zeros((rng.shape[0], 4), device=rng.device)
        state["renderer"].render(rng, pix, spp, depth)
        return {"pixels": pix, "states": rng}
    ds = state["scene"]
    pix = torch.zeros((rng.shape[0], 4), device=rng.device)
    ds.render(rng, pix, spp, depth)
    if case["scene"] == "gradient":
        # squared error against the target image, per accumulated sample
        dloss = (pix / spp - state["target"]) * (2.0 / spp)
        dloss[:, 3] = 0.0
        grad = torch.zeros((state["tex"].numel(), 4), device=rng.device)
        grad_env = torch.zeros((state["env_texels"], 4), device=rng.device)
        replay = state["states"].clone()
        ds.render_adjoint(replay, dloss, spp, depth, state["tex"], state["kind"], grad, state["env_tex"], grad_env)
        return {"pixels": pix, "states": rng, "grad": grad, "grad_env": grad_env, "replayed": replay}
    return {"pixels": pix, "states": rng, "image": postprocess.to_ldr(pix, ds.width, ds.height, spp)}


# ------------------------------------------------------------- work, exact


def _grid_vertices(n: int) -> int:
    side = max(2, math.ceil(math.sqrt(n / 2)) + 1)
    return side * side


def _ray_work(rays: int, tris: int) -> dict:
    """A ray passes at least one node per level of a balanced tree (two
    boxes, 15 operations each) and one triangle (50); the tree is read once
    where the rays between them reach all of it."""
    levels = math.log2(max(tris, 2))
    tree = min(112.0 * tris, rays * (64.0 * levels + 48.0))
    return {"bytes": tree, "flops": rays * (levels * 30.0 + 50.0)}


def work(case: dict) -> dict:
    family = case["family"]
    if family == "build":
        n = case["tris"]
        verts = 12 * _grid_vertices(n) + 12 * n if case["mesh"] == "grid" else 36 * n
        # vertices (and faces) in; a 64-byte node and a 48-byte record per triangle out
        return {"bytes": verts + 112 * n, "flops": 40 * n}
    if family == "build_batched":
        span = math.log(case["max_tris"] / case["min_tris"])
        n = int(case["scenes"] * (case["max_tris"] - case["min_tris"]) / span)  # mean of a log-uniform count
        return {"bytes": (36 + 112) * n, "flops": 40 * n}
    if family == "trace":
        w = _ray_work(case["rays"], case["tris"])
        w["bytes"] += (33 if case["query"] == "shadow" else 40) * case["rays"]
        return w
    if case["scene"] == "batch":
        span = math.log(case["max_tris"] / case["min_tris"])
        tris = case["scenes"] * (case["max_tris"] - case["min_tris"]) / span
        pixels = case["scenes"] * sum(r * r for r in batch.RESOLUTIONS) / len(batch.RESOLUTIONS)
        per_scene = tris / case["scenes"]
    else:
        pixels = case["width"] * case["height"]
        tris = per_scene = {"cornell": 996, "gradient": 996, "terrain": 2228224}[case["scene"]]
    samples = pixels * case["spp"]
    passes = 3 if case["scene"] == "gradient" else 1  # the image, then its paths once more with derivatives
    w = _ray_work(int(samples), int(per_scene))
    # per pixel: random state and sum read and written; the tree once
    return {"bytes": passes * 64.0 * pixels + 112.0 * tris, "flops": passes * (w["flops"] + 200.0 * samples)}


def exact(case: dict, seed: int):
    """The closest hit's distance by testing every triangle in 64 bits, for
    queries small enough; the other outputs are ids, bytes and random states
    or have no direct evaluation."""
    if case["family"] != "trace" or case["query"] != "closest" or case["rays"] * case["tris"] > 2e9:
        return None
    device = torch.device("cuda")
    vertices, faces, n = _mesh(case, seed, device)
    rays = _rays(case, seed, device).double()
    idx = faces.long() if faces is not None else torch.arange(3 * n, device=device).view(n, 3)
    v = torch.stack(vertices, -1).double()[idx]
    p0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    out = torch.empty(rays.shape[0], dtype=torch.float64, device=device)
    step = max(1, int(2e7 // n))
    for lo in range(0, rays.shape[0], step):
        o, tmax, d = rays[lo:lo + step, None, 0:3], rays[lo:lo + step, 3], rays[lo:lo + step, None, 4:7]
        p = torch.linalg.cross(d.expand(-1, n, -1), e2[None].expand(d.shape[0], -1, -1))
        det = (e1[None] * p).sum(-1)
        s = o - p0[None]
        b1 = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand(s.shape[0], -1, -1))
        b2 = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (det.abs() >= 1e-6) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= 0)
        best = torch.where(ok, t, math.inf).amin(-1)
        out[lo:lo + step] = torch.minimum(best, tmax)
    return {"id": None, "t": out}
