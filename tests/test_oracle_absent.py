"""Tests that call the reference library themselves are skipped, not failed,
where it is not built; other errors still fail."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
from oracle import ref

def test_calls_the_reference(monkeypatch):
    monkeypatch.setattr(ref, "_LIB", None)
    monkeypatch.setattr(ref, "REF_SO", "/nowhere/libref.so")
    ref.load()

def test_fails_on_its_own():
    raise RuntimeError("not the oracle")
"""


def test_missing_reference_library_skips(tmp_path):
    (tmp_path / "test_inner.py").write_text(BODY)
    p = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "tests.conftest", "-p", "no:cacheprovider",
                        str(tmp_path / "test_inner.py")], cwd=ROOT, capture_output=True, text=True)
    assert "1 failed, 1 skipped" in p.stdout, p.stdout
