"""The autotuner against untuned calls (needs a GB300): the default it times has the segment that an
untuned call of that size gets, and cache lines of another library version are passed over."""
import json

import numpy as np
import pytest

from katric_gb300 import Graph, _native

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def tune(counter, g, cache):
    fo = torch.from_numpy(g.first_out.view(np.int64).copy()).cuda()
    hd = torch.from_numpy(g.head.view(np.int32).copy()).cuda()
    conf, info = counter.autotune(fo.data_ptr(), hd.data_ptr(), g.n, g.nnz, cache_path=str(cache))
    return conf, info, [json.loads(line) for line in cache.read_text().splitlines()]


@pytest.mark.parametrize("edges,segment", [(1 << 10, 64), (1 << 16, 64), (450_000, 64), (600_000, 128),
                                           (1_100_000, 256), (4_400_000, 1024)])
def test_default_is_that_of_an_untuned_call(counter, tmp_path, edges, segment):
    """Adjacency slots per tile: the largest power of two that leaves 8192 tiles, within 64..1024."""
    g = Graph.gnm(1 << 15, edges, seed=3)
    conf, info, lines = tune(counter, g, tmp_path / "tune.jsonl")
    assert len(lines) == 1 and lines[0]["default_segment"] == segment
    assert info["ms"] <= info["default_ms"]
    # default, hybrid, three small bounds, two medium bounds, four segments and the tile order, at least
    assert conf.intersection_method != "auto" or info["candidates"] >= 12


def test_lines_of_another_version_are_passed_over(counter, tmp_path):
    g = Graph.gnm(4000, 30_000, seed=4)
    cache = tmp_path / "tune.jsonl"
    conf, info, lines = tune(counter, g, cache)
    assert not info["from_cache"] and lines[0]["version"] == _native.load().ktri_version().decode()
    old = dict(lines[0], version="katric_gb300 1.0 (sm_103a)", segment=1024, small_outdegree=7)
    none = {k: v for k, v in old.items() if k != "version"}
    cache.write_text("".join(json.dumps(x) + "\n" for x in (old, none)))
    conf, info, lines = tune(counter, g, cache)
    assert not info["from_cache"] and len(lines) == 3
    cache.write_text("".join(json.dumps(x) + "\n" for x in (lines[2], old, none)))
    again, info, lines = tune(counter, g, cache)
    assert info["from_cache"] and len(lines) == 3 and again == conf
