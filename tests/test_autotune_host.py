"""The autotuner's cache key: problems whose substeps run on another schedule do not share an entry."""

import json

from genesis_b200 import autotune


class _Problem:
    def __init__(self, n, eligible, n_blocks=5000):
        self.n, self.n_blocks, self.specs, self._eligible = n, n_blocks, [None], eligible
        self.applied = None

    def rotate_eligible(self):
        return self._eligible

    def retune(self, **kw):
        self.applied = kw


def test_key_tells_schedules_apart():
    # one power of two on both sides of the limit, and the same sizes with and without colliders
    assert autotune.signature(_Problem(290_000, True)) != autotune.signature(_Problem(310_000, False))
    assert autotune.signature(_Problem(20_000, True)) != autotune.signature(_Problem(20_000, False))
    assert autotune.signature(_Problem(20_000, True)) == autotune.signature(_Problem(20_001, True))


def test_entries_of_an_earlier_schedule_are_left_alone(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("GENESIS_B200_TUNE_CACHE", str(path))
    small = _Problem(20_000, True)
    earlier = "n32768_blk8192_inst1"  # the key before the schedule was part of it
    entry = lambda p: {"best": {"chunk_particles": p}, "times": {}}
    path.write_text(json.dumps({earlier: entry(256), autotune.signature(small): entry(128)}))
    candidates = {"grid_ctas": (0,)}  # (nothing is timed: the entry decides)
    assert autotune.tune(small, candidates)[0] == {"chunk_particles": 128} == small.applied
