"""Files of tuned launch geometry (CPU only)."""
import json


def test_files_of_segment_lengths_are_timed_again(tmp_path, monkeypatch):
    """A file from when the level-1 knob was a z-segment length in chunks: its level-1 entries would be read as
    blocks per SM, so they are left out; the others, and files saved now, load as they are."""
    from loadpath_b200 import tune

    monkeypatch.setattr(tune, "_RESULTS", {})
    old = {"fine_f32 128 64 64": {"best": 2, "us": {"0": 30.0, "1": 40.0, "2": 29.0}},
           "level1_f32 64 32 32": {"best": 1, "us": {"0": 20.0, "1": 19.0, "2": 20.0, "3": 22.0, "4": 23.0, "6": 25.0, "9": 30.0}}}
    path = str(tmp_path / "tuned.json")
    with open(path, "w") as fh:
        json.dump(old, fh)
    assert tune.load(path) == 2
    assert set(tune._RESULTS) == {("fine_f32", 128, 64, 64)}
    tune._RESULTS[("level1_f32", 64, 32, 32)] = {"best": 1, "us": {0: 20.0, 1: 19.0, 2: 20.0}}
    tune.save(path)
    want = dict(tune._RESULTS)
    tune._RESULTS.clear()
    assert tune.load(path) == 2 and tune._RESULTS == want


def test_candidates_keep_their_interface():
    from loadpath_b200 import tune

    assert tune.candidates(nchunks=9, lo=2) == [0, 2, 3, 4, 6, 9]
    assert tune.FINE_CANDIDATES == (0, 1, 2)
