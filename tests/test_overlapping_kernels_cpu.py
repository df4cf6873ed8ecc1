"""Kernels that start beside the kernel before them on the stream (programmatic dependent launch): what their source
must not do.  A kernel that is already resident while its inputs are still being written may read them only after its
wait, and only with coherent loads: non-coherent ones (``__ldg``, ``ld.global.nc``) are defined for memory that nothing
writes during the life of the kernel, and may hit a line that was cached before the write."""
import glob
import os
import re
import subprocess

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


def _overlapping_kernels():
    for path in FILES:
        code = _code(path)
        for m in re.finditer(r"__global__", code):
            start = code.index("\n{", m.end())
            if re.search(r"after_previous(<false>)?\(", code[start:code.index("\n}", start)]):
                signature = code[m.end():start]
                yield re.search(r"(\w+_kernel)\s*\(", signature).group(1), signature


def test_inputs_are_not_restrict():
    """``const T* __restrict__`` lets the compiler make the loads non-coherent and move them above the wait."""
    kernels = dict(_overlapping_kernels())
    assert len(kernels) >= 15
    assert [k for k, sig in kernels.items() if re.search(r"const\s+\w+\s*\*\s*__restrict__", sig)] == []


def test_no_spills_in_the_swiglu_quantiser(tmp_path):
    """The int32 form lives at the edge of its 64 registers: what the wait costs must not push it over."""
    from cannbench_operator_solutions_b200 import build

    cmd = [build._nvcc(), *build.NVCC_FLAGS, "-c", os.path.join(CSRC, "dqsq.cu"), "-o", str(tmp_path / "dqsq.o")]
    log = subprocess.run(cmd, check=True, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True).stdout
    spills = dict(re.findall(r"Compiling entry function '(\S*dqsq_rows_kernelILi0\S*)'.*?(\d+) bytes spill stores", log,
                             flags=re.S))
    assert {k: n for k, n in spills.items() if int(n) > 0} == {}
    # the forms that a call can reach: three of int32, four each of fp16 and bf16
    assert len(spills) == 3 and log.count("Compiling entry function") == 3 + 4 + 4 + 3


def test_next_kernel_is_let_in_after_the_wait_of_a_large_grid():
    """Let in ahead of the wait of a grid with more blocks than SMs, three kernels are resident at once and their blocks
    share the SMs unevenly."""
    code = _code(os.path.join(CSRC, "common.cuh"))
    steps = re.findall(r"if \((.* SMS)\)|griddepcontrol\.(\w+)", code)
    assert [a or b for a, b in steps] == ["BY_GRID && gridDim.x <= SMS", "launch_dependents", "wait",
                                          "!BY_GRID || gridDim.x > SMS", "launch_dependents"]


def test_registers_of_the_unvectorised_combine(tmp_path):
    """Three blocks of 256 threads per SM need 80 registers or fewer, without spills: the look-up of the next row stays
    with the vectorised form."""
    from cannbench_operator_solutions_b200 import build

    cmd = [build._nvcc(), *build.NVCC_FLAGS, "-c", os.path.join(CSRC, "ep.cu"), "-o", str(tmp_path / "ep.o")]
    log = subprocess.run(cmd, check=True, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True).stdout
    forms = re.findall(r"Compiling entry function '(\S*mfr_kernelILi[01]ELb0ELb0E\S*)'.*?(\d+) bytes spill stores"
                       r".*?Used (\d+) registers", log, flags=re.S)
    assert len(forms) == 4  # fp16 and bf16, 32- and 64-bit positions
    assert [f for f in forms if int(f[1]) > 0 or int(f[2]) > 80] == []
