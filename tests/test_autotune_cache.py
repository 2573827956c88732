"""The tuning cache: entries are found again, and entries of another candidate set are not."""
import json

import pytest

from spikesorting_fullpursuit_b200 import autotune


@pytest.fixture
def cache(tmp_path, monkeypatch):
    path = tmp_path / "tuning.json"
    monkeypatch.setenv("FBP_TUNE_CACHE", str(path))
    return path


def test_a_stored_entry_is_found(cache):
    best = {"lik_tiles": 0, "lik_group": 0, "lik_stages": 0, "pc_group": 4, "lik_epi": 0}
    assert autotune.cached(16, 40, 101, 100, "GPU") is None
    autotune._store(autotune.key_of(16, 40, 101, 100, "GPU"), best)
    assert autotune.cached(16, 40, 101, 100, "GPU") == best
    assert autotune.cached(16, 40, 101, 50, "GPU") is None
    assert autotune.cached(16, 40, 101, 100, "another GPU") is None


def test_entries_of_other_candidate_sets_are_measured_again(cache, monkeypatch):
    # as written before the library's own choice was a candidate
    old = {"lik_tiles": 0, "lik_group": 0, "lik_stages": 4, "pc_group": 8, "lik_epi": 2}
    cache.write_text(json.dumps({"C16-M40-W101-S100-GPU": old}))
    assert autotune.cached(16, 40, 101, 100, "GPU") is None
    autotune._store(autotune.key_of(16, 40, 101, 100, "GPU"), old)
    monkeypatch.setattr(autotune, "CANDIDATES", autotune.CANDIDATES + 1)
    assert autotune.cached(16, 40, 101, 100, "GPU") is None
