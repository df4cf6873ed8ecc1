"""Kernels that start beside the kernel before them on the stream (programmatic dependent launch): what their source
must not do.  A kernel that is already resident while its inputs are still being written may read them only after its
wait, and only with coherent loads: non-coherent ones (``__ldg``, ``ld.global.nc``) are defined for memory that nothing
writes during the life of the kernel, and may hit a line that was cached before the write."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cannbench_operator_solutions_b200",
                    "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _code(path):
    """The file without its comments."""
    with open(path) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_no_non_coherent_loads(path):
    assert not re.findall(r"__ldg\s*\(|ld\.global\.nc\S*", _code(path))
