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


def _bodies():
    for path in FILES:
        code = _code(path)
        for m in re.finditer(r"__global__", code):
            start = code.index("\n{", m.end())
            yield re.search(r"(\w+_kernel)\s*\(", code[m.end():start]).group(1), code[start:code.index("\n}", start)]


def test_kernels_beside_the_one_before_them_wait_at_their_end():
    """Whoever waits for such a kernel has then waited for both; its reads are behind a fence, not behind a wait."""
    code = _code(os.path.join(CSRC, "beside.cuh"))
    steps = re.findall(r"griddepcontrol\.\w+|fence\.\w+\.\w+", code)
    assert steps == ["griddepcontrol.launch_dependents", "fence.acq_rel.gpu", "griddepcontrol.wait"]
    kernels = {name: body for name, body in _bodies() if "beside_previous()" in body}
    assert sorted(kernels) == ["ardq_rows_kernel", "gemm_tc_kernel"]
    for body in kernels.values():
        assert body.count("beside_previous()") == body.count("previous_complete()") == 1
        assert body.index("beside_previous()") < body.index("previous_complete()")


def test_what_runs_before_a_kernel_beside_it_lets_it_in_after_its_own_wait():
    """A kernel beside the one before it does not wait at its start: all that came before the two must be complete when it is
    let in.  The route plan's last kernel in both of its forms, and the first of a grouped matmul's two launches."""
    bodies = dict(_bodies())
    assert "after_previous<false>()" in bodies["rp_rank_kernel"] and "after_previous()" not in bodies["rp_rank_kernel"]
    plan = _code(os.path.join(CSRC, "ep.cu")).split("int w8a8_route_plan(")[1].split("\n}")[0]
    forms = plan.split("RP_MAX_EXPERTS)")[1].split("return")[0].split("} else {")
    assert [re.findall(r"(rp_\w+_kernel)", form)[-1] for form in forms] == ["rp_rank_kernel", "rp_rank_kernel"]
    step = _code(os.path.join(CSRC, "moe_step.cu"))
    assert re.findall(r"rc = (\w+)\(", step.split("int one_rank_step(")[1])[:3] == [
        "w8a8_route_plan", "add_rms_norm_dynamic_quant_beside", "dispatch_rows_local"]
    assert step.count("_beside(") == 1  # nobody else asks for it
    # the matmul: FIRST waits, then lets the next in; SECOND is only ever launched behind FIRST
    assert re.search(r"order == ORDER_FIRST_OF_TWO\) \{\s*after_previous<false>\(\);\s*\} else if \(p\.order == ORDER_SECOND_OF_TWO\)"
                     r" \{\s*beside_previous\(\);", bodies["gemm_tc_kernel"])
    run = _code(os.path.join(CSRC, "gemm.cu")).split("static int run_grouped(")[1].split("\n}")[0]
    assert re.findall(r"ORDER_\w+", run) == ["ORDER_FIRST_OF_TWO", "ORDER_PLAIN", "ORDER_ALONE", "ORDER_SECOND_OF_TWO",
                                             "ORDER_ALONE"]
    assert run.count("overlap ? ORDER_") == 2
