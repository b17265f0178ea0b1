"""Without its harness the oracle's reference class fails; it does not skip
the test that asked for it."""
import unittest

import pytest


def test_missing_harness_is_an_error(monkeypatch, tmp_path):
    import oracle as O

    monkeypatch.setattr(O, "REF_PATH", str(tmp_path / "none.so"))
    with pytest.raises(FileNotFoundError) as e:
        O.Reference()
    assert not isinstance(e.value, unittest.SkipTest)
