"""Without the reference's kernels a caller sees a missing file, and a test
that needs them is skipped."""
import unittest

import pytest


def test_missing_kernels(monkeypatch, tmp_path):
    from oracle.ref_gpu import replay
    monkeypatch.setattr(replay, 'LIB', str(tmp_path / 'none.so'))
    monkeypatch.setattr(replay, '_lib', None)
    with pytest.raises(FileNotFoundError) as e:
        replay.load()
    assert isinstance(e.value, unittest.SkipTest)
