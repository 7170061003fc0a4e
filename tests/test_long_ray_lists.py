"""Ray lists whose counts reach the limits of 30- and 32-bit words.

A sort pass's look-back carries counts below 2^30 under two flag bits, and
rays of one origin all have one key, so lists of 2^30 rays and more are sorted
in parts.  The lists here repeat a few rays with a period that divides no power
of two: an answer taken from a wrong ray, or written to a wrong place, differs.
"""
import ctypes as C

import pytest
import torch

from clear_gb300 import _lib, lbvh
from clear_gb300 import workloads as W
from clear_gb300.build import build

PERIOD = 4099
STEP = 1 << 25


def _bytes(n: int) -> int:
    b = C.c_uint64(0)
    assert _lib.load().clr_trace_sort_workspace_bytes(C.c_uint32(n), C.byref(b)) == 0
    return b.value


def test_sorted_parts_share_a_workspace():
    build()
    most = _bytes((1 << 30) - 4096)
    assert _bytes((1 << 30) - 4097) <= most
    for n in ((1 << 30) - 4095, 1 << 30, (1 << 31) + 5, (1 << 32) - 1):
        assert _bytes(n) == most, n


def _long_list(cuda, n: int, one_origin: bool):
    """A small tree, PERIOD rays with their answers, and n rays repeating them."""
    free = torch.cuda.mem_get_info(cuda)[0]
    if free < 64 * n + (24 << 30):
        pytest.skip(f"{free >> 30} GiB of device memory free")
    tris = 64
    v = tuple(torch.from_numpy(a).to(cuda) for a in W.triangle_soup(tris, seed=3))
    bvh = lbvh.LBVHBuilder(tris, cuda).perform(v, None, tris, 10)
    few = torch.from_numpy(W.shadow_rays(PERIOD, seed=4)).to(cuda)
    if one_origin:
        few[:, 0:3] = torch.tensor([0.5, 0.5, 2.0], device=cuda)
        few[:, 3] = 3.0
        few[:, 4:7] -= torch.tensor([0.0, 0.0, 2.0], device=cuda)
    rays = torch.empty((n, 8), device=cuda)
    for lo in range(0, n, STEP):
        hi = min(n, lo + STEP)
        rays[lo:hi] = few[torch.arange(lo, hi, device=cuda) % PERIOD]
    return bvh, few, rays


def _repeats(got: torch.Tensor, few: torch.Tensor) -> bool:
    n = got.shape[0]
    for lo in range(0, n, STEP):
        hi = min(n, lo + STEP)
        if not torch.equal(got[lo:hi], few[torch.arange(lo, hi, device=got.device) % PERIOD]):
            return False
    return True


@pytest.mark.gpu
def test_sorted_lists_above_2_30_rays(cuda):
    n = (1 << 30) + 4099
    bvh, few, rays = _long_list(cuda, n, one_origin=True)
    want_id, want_t = lbvh.trace_closest(bvh, few, ordered=False)
    want_occ = lbvh.trace_shadow(bvh, few)
    assert 0 < int((want_id >= 0).sum()) < PERIOD  # some rays hit, some miss
    ids, ts = lbvh.trace_closest(bvh, rays, sort=True)
    assert _repeats(ids, want_id) and _repeats(ts.view(torch.int32), want_t.view(torch.int32))
    del ids, ts
    assert _repeats(lbvh.trace_shadow(bvh, rays, sort=True), want_occ)
    assert _lib.device_status() == 0
    del rays
    torch.cuda.empty_cache()


@pytest.mark.gpu
def test_lists_above_2_31_rays(cuda):
    """Ray r's record is floats 8 r to 8 r + 7: float4 2 r, beyond 32 bits here."""
    n = (1 << 31) + 4099
    bvh, few, rays = _long_list(cuda, n, one_origin=False)
    for ordered in (True, False):
        ids, ts = lbvh.trace_closest(bvh, rays, ordered=ordered)
        want_id, want_t = lbvh.trace_closest(bvh, few, ordered=ordered)
        assert _repeats(ids, want_id) and _repeats(ts.view(torch.int32), want_t.view(torch.int32)), ordered
        del ids, ts
    assert _repeats(lbvh.trace_shadow(bvh, rays), lbvh.trace_shadow(bvh, few))
    ids, counts = lbvh.trace_closest_counted(bvh, rays)
    want_id, want_counts = lbvh.trace_closest_counted(bvh, few)
    assert _repeats(ids, want_id) and _repeats(counts, want_counts)
    assert _lib.device_status() == 0
    del rays, ids, counts
    torch.cuda.empty_cache()
