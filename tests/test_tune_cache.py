"""The autotuner's cache and candidates, with the timing replaced: shapes timed
on other kernels are not taken from the cache, what the shapes depend on is in
the key, and no shape is timed that no kernel reads."""
import json
from types import SimpleNamespace

import numpy as np
import pytest

from imagestackalignator_b200 import params as P, tune


class Merger:
    def __init__(self, params):
        self.params, self.entries = params, None

    def set_tuning(self, entries=()):
        self.entries = list(entries)


@pytest.fixture
def timed(monkeypatch):
    """The entries that were timed; 16 rows a strip and blocks of 64 x 4 are the quickest."""
    log = []

    def cost(merger, item, entry, reps):
        log.append(entry)
        return 10.0 - 2.0 * (entry["lk_strip_rows"] == 16) - 2.0 * (entry.get("acc_block_x") == 64)

    monkeypatch.setattr(tune, "_time_merge", cost)
    monkeypatch.setattr(tune, "_device_name", lambda: "GPU")
    return log


def item(params, cfa=(0, 1, 1, 2), w=1024, h=768):
    return dict(raw=np.empty((3, h, w), np.uint16), info=SimpleNamespace(cfa=list(cfa)), params=params)


def test_entries_of_other_kernels_are_not_used(timed, tmp_path):
    """A cache as it was written before the key named the kernels."""
    path = tmp_path / "tuning.json"
    p = P.MergeParams(merge_scale=1.5)
    path.write_text(json.dumps({f"GPU|{tune.burst_class(1024, 768, 1.5)}": dict(lk_strip_rows=128, acc_block_x=16, acc_block_y=16)}))
    e = tune.tune(Merger(p), [item(p)], cache_path=str(path))
    assert timed and e == [dict(width=1024, height=768, lk_strip_rows=16, acc_block_x=64, acc_block_y=4)]
    n = len(timed)
    assert tune.tune(Merger(p), [item(p)], cache_path=str(path)) == e and len(timed) == n  # from the cache
    q = P.MergeParams(merge_scale=1.5, window_size_lk=21)
    tune.tune(Merger(q), [item(q)], cache_path=str(path))
    assert len(timed) > n  # another window, other strips


@pytest.mark.parametrize("params,cfa,reads", [
    (dict(merge_scale=2.0), (0, 1, 1, 2), False), (dict(merge_scale=1.0), (1, 2, 0, 1), False), (dict(), (2, 1, 1, 0), False),
    (dict(super_resolution=True), (1, 0, 2, 1), False), (dict(merge_scale=1.5), (0, 1, 1, 2), True), (dict(merge_scale=3.0), (0, 1, 1, 2), True),
    (dict(merge_scale=2.0, sample_mode=P.SAMPLE_BILINEAR), (0, 1, 1, 2), True), (dict(merge_scale=2.0), (1, 1, 1, 1), True)])
def test_blocks_are_timed_only_where_they_are_read(timed, tmp_path, params, cfa, reads):
    p = P.MergeParams(**params)
    e = tune.tune(Merger(p), [item(p, cfa)], cache_path=str(tmp_path / "t.json"))
    assert any(t.get("acc_block_x") for t in timed) == reads
    assert (e[0]["acc_block_x"] == 64) == reads


def test_strip_heights_reach_the_short_strips():
    """Small frames run strips of 8 to 24 rows by the library's own choice."""
    assert {8, 16, 24} <= set(tune.LK_ROWS)


def test_contexts_side_by_side_have_entries_of_their_own(timed, tmp_path, monkeypatch):
    """Shapes of a batch are timed on all its contexts, and kept apart from those of a burst alone."""
    seen = []
    monkeypatch.setattr(tune, "_time_merge", lambda merger, item, entry, reps, beside=(): seen.append(len(beside)) or
                        10.0 + (entry["lk_strip_rows"] == 16 and len(beside)) - 2.0 * (entry["lk_strip_rows"] == 16 and not beside))
    p, path = P.MergeParams(merge_scale=2.0), str(tmp_path / "t.json")
    m, others = Merger(p), [Merger(p), Merger(p)]
    assert tune.tune(m, [item(p)], cache_path=path)[0]["lk_strip_rows"] == 16
    assert tune.tune(m, [item(p)], cache_path=path, beside=others)[0]["lk_strip_rows"] == 0
    assert set(seen) == {0, 2} and len(json.loads(open(path).read())) == 2
    assert all(x.entries == [] for x in [m, *others])
