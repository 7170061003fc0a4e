"""Scratch and routes of the batched build over calls with different splits.

The scratch of a builder depends on its capacity and the largest number of
scenes so far, not on how the triangles are split among them: a call of a warm
builder allocates nothing, so it can be captured, and a captured build's
scratch stays where it is."""
import ctypes as C

import numpy as np
import pytest
import torch

from clear_gb300 import _lib, lbvh
from clear_gb300 import workloads as W

pytestmark = pytest.mark.gpu

EVEN = [4096] * 16
UNEVEN = [1, 8191] * 8  # as many triangles and scenes, more tiles of 4,096 keys


def _offsets(sizes):
    return [int(o) for o in np.concatenate([[0], np.cumsum(sizes)])]


def _build(builder, v, b):
    """Into the buffers of `b`; the offsets array is returned to be kept alive."""
    offs = (C.c_uint32 * len(b.offsets))(*b.offsets)
    _lib.call("clr_lbvh_build_batched", builder._h, v[0].data_ptr(), v[1].data_ptr(), v[2].data_ptr(), None, offs,
              len(b), b.bits, 8, b.nodes.data_ptr(), b.tris.data_ptr(), b.root_boxes.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    return offs


@pytest.mark.parametrize("bits", [10, 20])
def test_warm_builds_of_another_split_are_captured(cuda, bits):
    n = sum(EVEN)
    assert sum(UNEVEN) == n
    v = tuple(torch.from_numpy(a).to(cuda) for a in W.triangle_soup(n, seed=11))
    want = lbvh.LBVHBuilder(n, cuda).perform_batched(v, None, _offsets(UNEVEN), bits)
    builder = lbvh.LBVHBuilder(n, cuda)
    even, uneven = (lbvh.BatchBVH(_offsets(s), bits, cuda) for s in (EVEN, UNEVEN))
    _build(builder, v, even)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        keep = _build(builder, v, uneven)
    _build(builder, v, even)  # between the capture and its replay
    graph.replay()
    torch.cuda.synchronize()
    assert len(keep) == len(UNEVEN) + 1 and _lib.device_status() == 0
    for s, size in enumerate(UNEVEN):
        a, b = uneven.scene(s), want.scene(s)
        assert torch.equal(a.tris, b.tris) and torch.equal(a.root_box.view(torch.int32), b.root_box.view(torch.int32))
        used = (size - 1) * _lib.NODE_BYTES
        assert torch.equal(a.nodes[:used], b.nodes[:used])
