"""The autotuner and batches searched over block pools: the trace block reaches no
search kernel there, so it is not timed and stays at its default."""
import pytest

from clear_gb300 import autotune
from test_autotune import FakeBatch, _patch


@pytest.mark.parametrize("pools", [False, True])
def test_trace_block_is_timed_where_it_counts(monkeypatch, tmp_path, pools):
    calls = []
    _patch(monkeypatch, tmp_path, calls)
    br = FakeBatch()
    br.pool_searches = pools
    autotune.tune(br, max_depth=5)
    renders = [c for kind, c in calls if kind == "render"]
    timed = len(autotune.POOL_CANDIDATES) + len(autotune.SHADE_BLOCKS) + (0 if pools else len(autotune.TRACE_BLOCKS))
    assert len(renders) == timed
    assert {c["trace_block"] for c in renders} == ({128} if pools else set(autotune.TRACE_BLOCKS))
    assert br.config() == {"trace_block": 128 if pools else 64, "shade_block": 96, "pool_slots": 2 << 20}


@pytest.mark.gpu
def test_batches_say_whether_pools_search_them(cuda, monkeypatch):
    from clear_gb300.batch import BatchRenderer, random_scene
    from test_megakernel_search_gpu import _with_cutouts

    plain = [random_scene(n, 16, 16, n) for n in (50, 60)]
    cut = _with_cutouts(lambda: random_scene(70, 16, 16, 7), monkeypatch)
    assert BatchRenderer(plain, cuda).pool_searches
    assert not BatchRenderer(plain + [cut], cuda).pool_searches
