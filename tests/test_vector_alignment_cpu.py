"""Per-channel vectors of the matmuls are read in 16-byte pieces: one that starts elsewhere (a contiguous view at an odd
offset) is refused before anything is launched; a single value may lie wherever its type may."""
import ctypes

import pytest

from cannbench_operator_solutions_b200 import _lib as L


@pytest.fixture(scope="module")
def lib():
    from cannbench_operator_solutions_b200 import build

    build.build_library()
    return L.load()


def _address():
    buf = (ctypes.c_char * 8192)()
    return buf, (ctypes.addressof(buf) + 255) & ~255


BIAS = {"i32": L.QM_BIAS_I32, "f16": L.QM_BIAS_F16, "bf16": L.QM_BIAS_BF16, "f32": L.QM_BIAS_F32}


# (what lies off, its flags, by how many bytes)
@pytest.mark.parametrize("which,flags,off", [
    ("scale", L.QM_SCALE_PERCHAN, 4), ("scale", L.QM_SCALE_PERCHAN, 8), ("scale", L.QM_SCALE_PERCHAN | L.QM_SCALE_BF16, 2),
    ("scale", L.QM_SCALE_PERCHAN | L.QM_SCALE_BF16, 14), ("offset", L.QM_HAS_OFFSET | L.QM_OFFSET_PERCHAN, 4),
    *[("bias", (k << L.QM_BIAS_SHIFT) | L.QM_BIAS_PERCHAN, 4 if n in ("i32", "f32") else 2) for n, k in BIAS.items()],
    # single values: only their own type's alignment counts
    ("scale", 0, 1), ("scale", 0, 2), ("scale", L.QM_SCALE_BF16, 1), ("offset", L.QM_HAS_OFFSET, 2), ("pertoken", L.QM_HAS_PT, 2),
    *[("bias", k << L.QM_BIAS_SHIFT, 2 if n in ("i32", "f32") else 1) for n, k in BIAS.items()],
])
def test_quant_matmul(lib, which, flags, off):
    keep, p = _address()
    at = {name: p + (off if name == which else 0) for name in ("scale", "offset", "pertoken", "bias")}
    assert lib.w8a8_quant_matmul(p, p, at["scale"], at["offset"], at["pertoken"], at["bias"], p, 1, 16, 32, 32, flags, L.DT_BF16,
                                 L.W_KN, 0, None) == L.ERR_ALIGN


@pytest.mark.parametrize("kind,stride", [(L.QM_BIAS_F16, 4), (L.QM_BIAS_BF16, 33), (L.QM_BIAS_F32, 2), (L.QM_BIAS_I32, 1)])
def test_quant_matmul_bias_of_each_batch(lib, kind, stride):
    keep, p = _address()
    flags = (kind << L.QM_BIAS_SHIFT) | L.QM_BIAS_PERCHAN | L.QM_PT_MOD_M
    assert lib.w8a8_quant_matmul(p, p, p, None, None, p, p, 2, 16, 32, 32, flags, L.DT_BF16, L.W_KN, stride, None) == L.ERR_ALIGN


@pytest.mark.parametrize("dtype,w_off,x_off,bias_dtype,bias_off", [
    (L.DT_I8, 4, 0, None, 0), (L.DT_I8, 8, 0, None, 0), (L.DT_I8, 0, 2, None, 0), (L.DT_I8, 0, 0, L.DT_F32, 4),
    (L.DT_I8, 0, 0, L.DT_BF16, 2), (L.DT_BF16, 0, 0, L.DT_BF16, 8), (L.DT_F16, 0, 0, L.DT_F16, 2), (L.DT_F16, 0, 0, L.DT_F32, 12),
    (L.DT_F32, 0, 0, L.DT_F32, 4)])
@pytest.mark.parametrize("to_rows", [False, True])
def test_grouped_matmul(lib, dtype, w_off, x_off, bias_dtype, bias_off, to_rows):
    if to_rows and dtype == L.DT_F32:
        pytest.skip("fp32 results are not stored by row addresses")
    keep, p = _address()
    ends = (ctypes.c_int64 * 2)(3, 8)
    quantised = dtype == L.DT_I8
    call = lib.w8a8_grouped_matmul_to_rows if to_rows else lib.w8a8_grouped_matmul
    rc = call(p, p, None if bias_dtype is None else p + bias_off, p, p + x_off if quantised else None,
              p + w_off if quantised else None, 8, 64, 32, 2, ends, 0, dtype, dtype if bias_dtype is None else bias_dtype,
              L.DT_BF16 if quantised else dtype, L.W_KN, p, 1 << 30, None)
    assert rc == L.ERR_ALIGN


def test_grouped_matmul_swiglu_quant(lib):
    keep, p = _address()
    ends = (ctypes.c_int64 * 2)(3, 8)
    for w_off, x_off, s_off in ((4, 0, 0), (0, 2, 0), (0, 0, 2)):
        assert lib.w8a8_grouped_matmul_swiglu_quant(p, p, p + w_off, p + x_off, p, p + s_off, 8, 32, 64, 2, ends, 0, L.W_KN, 0, p,
                                                    1 << 30, None) == L.ERR_ALIGN
