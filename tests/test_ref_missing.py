"""Tests that compare with the reference's own library are skipped where it was
not built; other errors stay errors."""

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

INNER = """
import pytest
from oracle import ref


def test_needs_the_library(monkeypatch):
    monkeypatch.setattr(ref, "_lib", None)
    monkeypatch.setattr(ref, "REF_SO", "/nonexistent/libimate_ref.so")
    ref.load()


def test_needs_the_gpu_library(monkeypatch):
    monkeypatch.setattr(ref, "_gpu_lib", None)
    monkeypatch.setattr(ref, "REF_GPU_SO", "/nonexistent/libimate_ref_gpu.so")
    ref.load_gpu()


def test_another_missing_file():
    open("/nonexistent/file")
"""


def test_a_library_that_was_not_built_skips(tmp_path):
    (tmp_path / "test_inner.py").write_text(INNER)
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(
        [HERE, os.path.dirname(HERE), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run(
        [sys.executable, "-m", "pytest", "-q", "-rA", "-p", "conftest",
         "-p", "no:cacheprovider", str(tmp_path / "test_inner.py")],
        cwd=str(tmp_path), env=env, capture_output=True, text=True)
    assert "2 skipped" in r.stdout and "1 failed" in r.stdout, r.stdout
    assert "test_another_missing_file" in r.stdout
