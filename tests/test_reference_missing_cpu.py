"""Where the reference's CPU code is not built, the tests that need it as a
checker are skipped with that reason; a check that fails before, or any other
error, still fails."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

TESTS = """
from oracle import build_ref, ref

build_ref.available = lambda: False
build_ref.LIB = "/nonexistent/libref.so"
ref._lib = None


def test_needs_the_checker():
    ref.lib()


def test_fails_before_the_checker():
    assert False
    ref.lib()


def test_other_error():
    raise RuntimeError("another error")


def test_passes():
    assert not ref.available()
"""


def test_missing_checker_is_skipped(tmp_path):
    (tmp_path / "conftest.py").write_text("from tests.conftest import pytest_runtest_call\n")
    (tmp_path / "test_inner.py").write_text(TESTS)
    run = subprocess.run([sys.executable, "-m", "pytest", "-q", "-rs", "-p", "no:cacheprovider", str(tmp_path)],
                         capture_output=True, text=True, cwd=ROOT, env={**os.environ, "PYTHONPATH": ROOT})
    assert "2 failed, 1 passed, 1 skipped" in run.stdout, run.stdout + run.stderr
    assert "libref.so is not built" in run.stdout
