"""The BRIEF table where no reference checkout and no table of the user's is
at hand: load() refuses, the tests, smoke check and benchmark take the seeded
stand-in and name it."""
import numpy as np
import pytest

from uni_slam_gb300 import pattern


def test_stand_in(tmp_path, monkeypatch):
    monkeypatch.delenv("USLAM_BRIEF_PATTERN", raising=False)
    monkeypatch.setattr(pattern, "STAGED", str(tmp_path / "absent.txt"))
    with pytest.raises(FileNotFoundError):
        pattern.load(pattern.STAGED)
    got, source = pattern.load_or_stand_in()
    assert got.dtype == np.int32 and got.shape == (256, 4) and got.flags.c_contiguous and "stand-in" in source
    assert np.abs(got).max() == 13 and got[0].tolist() == [13, 13, -13, -13]
    assert np.array_equal(got, pattern.stand_in())


def test_a_users_table_comes_first(tmp_path, monkeypatch):
    own = np.arange(1024, dtype=np.int32).reshape(256, 4) % 9 - 4
    path = tmp_path / "own.txt"
    np.savetxt(path, own, fmt="%d")
    monkeypatch.setenv("USLAM_BRIEF_PATTERN", str(path))
    got, source = pattern.load_or_stand_in()
    assert np.array_equal(got, own) and str(path) in source
    # one that is named but missing is an error, not the stand-in
    monkeypatch.setenv("USLAM_BRIEF_PATTERN", str(tmp_path / "absent.txt"))
    with pytest.raises(FileNotFoundError):
        pattern.load_or_stand_in()
