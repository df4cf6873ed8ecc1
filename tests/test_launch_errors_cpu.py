"""A launch that fails is reported by the entry point and by nobody else: the error does not stay in the thread's
last-error slot, where the next library to look would take it for its own.  The failing launch is a fake: a library put
in front of the CUDA runtime whose every launch returns an error."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
static int last = 0;
static int fail(void) { return last = 9; /* cudaErrorInvalidConfiguration */ }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int dev) { (void)attr; (void)dev; *v = 148; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, unsigned long smem,
                                                           unsigned flags)
{ (void)f; (void)threads; (void)smem; (void)flags; *n = 4; return 0; }
int cudaLaunchKernelExC(const void* cfg, const void* f, void** args) { (void)cfg; (void)f; (void)args; return fail(); }
int cudaGetLastError(void) { int e = last; last = 0; return e; }
int cudaPeekAtLastError(void) { return last; }
"""

CALLS = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import importlib.util
spec = importlib.util.spec_from_file_location("L", sys.argv[1] + "/cannbench_operator_solutions_b200/_lib.py")
L = importlib.util.module_from_spec(spec); spec.loader.exec_module(L)
lib = L.load()
fake = ctypes.CDLL(sys.argv[2])
buf = (ctypes.c_char * 65536)()
p = (ctypes.addressof(buf) + 255) & ~255
calls = {
    "dynamic_quant": lambda: lib.w8a8_dynamic_quant(p, p, p, 4, 64, L.DT_BF16, 0, None),
    "norm": lambda: lib.w8a8_add_rms_norm_dynamic_quant(p, p, p, p, p, p, 4, 64, 1e-6, L.DT_BF16, 0, None),
    "gating": lambda: lib.w8a8_moe_gating_top_k_softmax(p, None, p, p, p, 4, 8, 2, L.DT_BF16, None),
    "swiglu": lambda: lib.w8a8_dequant_swiglu_quant(p, None, None, None, p, p, 4, 64, L.DT_BF16, 1, 0, None),
    "finalize": lambda: lib.w8a8_moe_finalize_routing(p, p, None, None, None, None, None, p, 4, 64, 2, 0, 8, 0,
                                                      L.DT_BF16, L.DT_BF16, None),
    "route_plan": lambda: lib.w8a8_route_plan(p, 4, 2, 8, p, p, p, p, 1 << 15, None),
}
for name, call in calls.items():
    assert call() == L.ERR_CUDA, name
    assert fake.cudaPeekAtLastError() == 0, name
print("reported once", len(calls))
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs a C compiler")
def test_failed_launch_leaves_no_error_behind(tmp_path):
    from cannbench_operator_solutions_b200 import build

    build.build_library()
    (tmp_path / "fake.c").write_text(FAKE)
    (tmp_path / "calls.py").write_text(CALLS)
    fake = str(tmp_path / "libfake.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", fake, str(tmp_path / "fake.c")], check=True)
    out = subprocess.run([sys.executable, str(tmp_path / "calls.py"), ROOT, fake], env={**os.environ, "LD_PRELOAD": fake},
                         stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert out.returncode == 0 and "reported once 6" in out.stdout, out.stdout
