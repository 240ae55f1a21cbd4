"""Where the reference oracle is not built, tests and fixtures that ask for it are skipped, and nothing else is."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

INNER = """
import oracle
import pytest

oracle.ref_lib_path = lambda timing=False: "/nonexistent/libebgref.so"
oracle._ref_cache = oracle._ref_timing_cache = None

@pytest.fixture
def mesh():
    return oracle.ref()

def test_in_the_body():
    oracle.ref()

def test_in_a_fixture(mesh):
    pass

def test_another_missing_file():
    with pytest.raises(FileNotFoundError):
        open("/nonexistent/file")

def test_other_errors_stay():
    open("/nonexistent/file")
"""


def test_missing_reference_skips(tmp_path):
    path = tmp_path / "test_inner.py"
    path.write_text(INNER)
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([HERE, os.path.dirname(HERE)]))
    out = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "conftest", "-p", "no:cacheprovider",
                          f"--rootdir={tmp_path}", str(path)], env=env, cwd=tmp_path, capture_output=True, text=True)
    assert "1 failed, 1 passed, 2 skipped" in out.stdout, out.stdout
