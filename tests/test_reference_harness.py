"""Tests that need the reference's compiled code are skipped where it cannot be
had (no HPMC source tree), and fail where it could have been built."""
from __future__ import annotations

import pytest

from tests import conftest


def _outcome(oracle):
    """What the test hook makes of a test that asks for the harness."""
    hook = conftest.pytest_runtest_call(None)
    next(hook)
    try:
        oracle.ref()
    except Exception as e:
        hook.throw(e)


@pytest.mark.parametrize("tree", [False, True])
def test_missing_harness(oracle, monkeypatch, tmp_path, tree):
    monkeypatch.setattr(oracle, "_REF_DIR", str(tmp_path))
    monkeypatch.setattr(oracle, "_ref", None)
    monkeypatch.setenv("HPMC_SRC", str(tmp_path))
    if tree:
        (tmp_path / "hpmc" / "src").mkdir(parents=True)
        (tmp_path / "hpmc" / "src" / "tables.cpp").touch()
    with pytest.raises(RuntimeError if tree else pytest.skip.Exception, match="reference harness not built"):
        _outcome(oracle)
