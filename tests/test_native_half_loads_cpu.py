"""ops.py without its native half: silent where that has not been built (as while building), a warning where it has been
built and does not load - every call would take longer, and nothing else would say so."""
import os
import subprocess
import sys

import pytest

PACKAGE = "cannbench_operator_solutions_b200"
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("built", [False, True])
def test_import(tmp_path, built):
    copy = tmp_path / PACKAGE
    copy.mkdir()
    source = os.path.join(ROOT, PACKAGE)
    for name in os.listdir(source):
        if name.endswith(".py"):
            os.symlink(os.path.join(source, name), copy / name)
    if built:
        (copy / "_calls.so").write_bytes(b"not a library")
    run = subprocess.run([sys.executable, "-W", "always", "-c", f"from {PACKAGE} import ops; print(ops.__file__, ops._calls)"],
                         cwd=tmp_path, capture_output=True, text=True, check=True)
    assert run.stdout.split() == [str(copy / "ops.py"), "None"]
    assert ("RuntimeWarning" in run.stderr and "_calls.so" in run.stderr) == built
