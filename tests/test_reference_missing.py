"""Tests that call the reference's own library are skipped where it is not built, as those are that ask first."""
import unittest

import numpy as np
import pytest


def test_calling_the_missing_reference_skips(monkeypatch):
    from oracle import ref
    monkeypatch.setattr(ref, "LIB_PATH", "/nonexistent/libqcbc_ref.so")
    monkeypatch.setattr(ref, "_lib", None)
    assert not ref.available()
    with pytest.raises(unittest.SkipTest):
        ref.condition(np.zeros(16), 1.0)
    with pytest.raises(FileNotFoundError):
        ref.lib()
