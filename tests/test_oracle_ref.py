"""A test that needs the reference library where its sources are absent is skipped: one
such failure would end a run that stops at the first."""
from __future__ import annotations

import numpy as np
import pytest


def test_absent_reference_skips(O, monkeypatch):
    import unittest
    monkeypatch.setattr(O._build, "build_ref", lambda *a, **k: None)
    monkeypatch.delitem(O._LIBS, "ref", raising=False)
    assert not O.ref_available()
    f = np.zeros((3, 3, 3), np.float32, order="F")
    with pytest.raises(unittest.SkipTest) as e:
        O.pull_affine(f, np.eye(4, dtype=np.float32), (3, 3, 3), O.Sett.make(1, 1, 1), kind="ref")
    assert isinstance(e.value, RuntimeError) and "absent" in str(e.value)


def test_this_is_reported_as_skipped(pytester_run):
    assert pytester_run["skipped"] == 1 and pytester_run["failed"] == 0


@pytest.fixture
def pytester_run(tmp_path):
    """A run of its own of one test that raises it."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    f = tmp_path / "test_needs_ref.py"
    f.write_text("import sys\nsys.path.insert(0, %r)\nfrom oracle.oracle import ReferenceUnavailable\n\n\n"
                 "def test_needs_it():\n    raise ReferenceUnavailable('absent')\n" % root)
    out = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "no:cacheprovider", str(f)], capture_output=True,
                         text=True, cwd=tmp_path).stdout
    return {k: int(n) for n, k in __import__("re").findall(r"(\d+) (passed|failed|skipped)", out)} | {
        k: 0 for k in ("passed", "failed", "skipped") if k not in out}
