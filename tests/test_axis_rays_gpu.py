"""Rays with zero direction components against the oracle (bit-exact ids,
distances and occlusion flags): parallel to one axis, to a coordinate plane, and
the zero direction, with components of both signs of zero; origins between,
beyond, exactly on and one step off the box planes; scenes and directions scaled
over the range in which boxes are classified, and past its ends."""
import numpy as np
import pytest
import torch

import oracle
from clear_gb300 import _lib, lbvh
from clear_gb300 import workloads as W
from test_ray_edges_gpu import _bricks

pytestmark = pytest.mark.gpu

RAYS = 24_000


def _rays(v, seed: int, dscale: float) -> np.ndarray:
    rng = np.random.default_rng(seed)
    p = np.stack(v, 1)
    lo, hi = p.min(0), p.max(0)
    ext = hi - lo
    o = rng.uniform(lo - 0.5 * ext, hi + 0.5 * ext, size=(RAYS, 3)).astype(np.float32)
    on = rng.random((RAYS, 3))
    plane = p[rng.integers(0, len(p), RAYS)]
    o = np.where(on < 0.4, plane, o)
    o = np.where(on < 0.2, np.nextafter(o, np.where(on < 0.1, np.inf, -np.inf).astype(np.float32)), o)
    d = rng.standard_normal((RAYS, 3))
    zeros = rng.integers(1, 4, RAYS)  # this many components
    zeros[rng.random(RAYS) < 0.45] = 2
    order = rng.permuted(np.tile(np.arange(3), (RAYS, 1)), axis=1)
    for k in range(3):
        d[np.arange(RAYS)[zeros > k], order[zeros > k, k]] = 0.0
    tiny = rng.random(RAYS) < 0.1  # a second component next to zero
    d[tiny] *= rng.choice([1.0, 1e-7, 1e-12], (int(tiny.sum()), 3))
    d = (d * dscale).astype(np.float32)
    d = np.where((d == 0) & (rng.random((RAYS, 3)) < 0.5), np.float32(-0.0), d)
    reach = float(ext.max()) / dscale
    tmax = np.where(rng.random(RAYS) < 0.5, np.inf, rng.choice([0.0, 0.25, 0.5, 1.0], RAYS) * reach)
    return W.pack_rays(o.astype(np.float32), d, tmax.astype(np.float32))


@pytest.mark.parametrize("dscale", [1.0, 2.0 ** -38, 2.0 ** 38, 2.0 ** 42])
@pytest.mark.parametrize("scene,scale", [("bricks", 1.0), ("bricks", 2.0 ** -12), ("bricks", 2.0 ** 30),
                                         ("soup", 1.0), ("soup", 2.0 ** 20), ("flat", 1.0)])
def test_axis_parallel_rays_match_oracle(cuda, scene, scale, dscale):
    v = _bricks(4) if scene != "soup" else W.triangle_soup(3000, seed=21)
    v = [a * np.float32(scale) for a in v]
    if scene == "flat":  # every box flat in y, several heights
        v[1] = np.repeat(v[1].reshape(-1, 3)[:, :1], 3, axis=1).reshape(-1)
    v = tuple(np.ascontiguousarray(a, dtype=np.float32) for a in v)
    n = len(v[0]) // 3
    bvh = lbvh.LBVHBuilder(n, cuda).perform(tuple(torch.from_numpy(a).to(cuda) for a in v), None, n, 10)
    ob = oracle.lbvh_build(*v, None, n, 10)
    rays = _rays(v, seed=n, dscale=dscale)
    r = torch.from_numpy(rays).to(cuda)
    want_id, want_t = oracle.trace_closest(*v, None, ob, rays)
    want_occ = oracle.trace_shadow(*v, None, ob, rays)
    for kw in ({"ordered": False}, {"ordered": True}, {"sort": True}):
        ids, ts = lbvh.trace_closest(bvh, r, **kw)
        np.testing.assert_array_equal(ids.cpu().numpy().view(np.uint32), want_id)
        np.testing.assert_array_equal(ts.cpu().numpy(), want_t)
    for sort in (False, True):
        np.testing.assert_array_equal(lbvh.trace_shadow(bvh, r, sort=sort).cpu().numpy(), want_occ)
    if dscale == 1.0 and scale == 1.0:
        assert (want_id != 0xFFFFFFFF).any()
    assert _lib.device_status() == 0
