"""ops.py's native half (calls in their plain form) against its Python half: the same outputs, bit for bit, with the same
shapes, strides and types; and the calls that it has to leave to the Python half."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs():
    g = torch.Generator(device="cuda").manual_seed(3)

    def f(*shape, dtype=torch.float32):
        return torch.randn(shape, generator=g, device="cuda").to(dtype)

    def i8(*shape):
        return torch.randint(-127, 128, shape, generator=g, device="cuda", dtype=torch.int8)

    bf, ends = torch.bfloat16, [3, 3, 20, 33]
    dev = torch.tensor(ends, device="cuda")
    i32 = (f(9, 64) * 1e4).int()
    counts = torch.tensor([[2, 1], [0, 4]], device="cuda")
    pos = torch.randperm(14, generator=g, device="cuda").int()
    yield "dynamic_quant", (f(5, 7, 40, dtype=bf),), {}
    yield "dynamic_quant", (f(1, 33, dtype=torch.float16),), {"round_direct": True}
    yield "dynamic_quant", (f(3, 64, dtype=bf).as_strided((1, 64), (128, 1)),), {}  # dense with an odd stride
    yield "add_rms_norm_dynamic_quant", (f(6, 48, dtype=bf), f(6, 48, dtype=bf), f(48, dtype=bf), 1e-6), {}
    yield "add_rms_norm_dynamic_quant", (f(48, dtype=bf), f(48, dtype=bf), f(48, dtype=bf), 1e-5), {"round_direct": True}
    yield "quant_matmul", (i8(5, 32), i8(32, 48), f(48)), {}
    yield "quant_matmul", (i8(5, 32), i8(48, 32), f(1)), {"transpose_x2": True, "output_dtype": "bfloat16"}
    yield "quant_matmul", (i8(2, 5, 32), i8(2, 32, 48), f(48, dtype=bf)), {
        "offset": f(48), "pertoken_scale": f(5), "bias": f(2, 1, 48, dtype=bf), "output_dtype": "float16"}
    yield "quant_matmul", (i8(5, 32), i8(32, 48), f(48)), {"bias": f(48).int(), "offset": f(1)}
    yield "grouped_matmul_swiglu_quant", (i8(33, 32), i8(4, 32, 64), f(4, 64), f(33), ends), {}
    yield "grouped_matmul_swiglu_quant", (i8(33, 32), i8(4, 64, 32), f(4, 64), f(33), dev), {"transpose_weight": True}
    for split in (0, 2, 3):
        yield "grouped_matmul", (f(33, 32, dtype=bf), f(4, 32, 48, dtype=bf), tuple(ends), f(4, 48, dtype=bf), split), {}
    yield "grouped_matmul", (f(33, 32), f(4, 32, 48), ends, None, 3), {}
    yield "grouped_matmul", (i8(33, 32), i8(4, 32, 48), dev, None, 3), {"x_scale": f(33), "weight_scale": f(4, 48)}
    yield "grouped_matmul", (i8(33, 32), i8(4, 32, 48), ends, f(4, 48), 3), {
        "x_scale": f(33), "weight_scale": f(4, 48), "output_dtype": torch.float16}
    yield "moe_re_routing", (i8(7, 48), counts, f(7)), {}
    yield "moe_re_routing", (f(7, 24, dtype=bf), counts.int(), f(7)), {"idx_type": 0}
    yield "moe_finalize_routing", (f(14, 24, dtype=bf), pos, f(7, 24, dtype=bf), None, None, f(7, 2)), {}
    yield "moe_finalize_routing", (f(14, 24), pos, f(7, 24), f(7, 24), f(3, 24), f(7, 2), torch.zeros_like(pos), 2), {}
    yield "moe_gating_top_k_softmax", (f(3, 5, 16, dtype=bf), None, 4), {}
    yield "moe_gating_top_k_softmax", (f(5, 60), torch.tensor([True, False, True, False, False], device="cuda"), 3), {}
    yield "dequant_swiglu_quant", (i32, f(64), f(9), f(32), True), {}
    yield "dequant_swiglu_quant", (f(9, 64, dtype=bf),), {"activate_left": False, "round_direct": True}


def _flat(v):
    return list(v) if isinstance(v, (tuple, list)) else [v]


def test_same_results(ops, monkeypatch):
    native = ops._calls
    assert native is not None
    for name, args, kwargs in _inputs():
        with_native = _flat(getattr(ops, name)(*args, **kwargs))
        monkeypatch.setattr(ops, "_calls", None)
        without = _flat(getattr(ops, name)(*args, **kwargs))
        monkeypatch.setattr(ops, "_calls", native)
        assert len(with_native) == len(without)
        for a, b in zip(with_native, without):
            assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride(), (name, a.stride(), b.stride())
            if a.dim() == 1 and a.dtype == torch.float32 and name == "moe_re_routing" and len(args) < 3:
                continue  # without scales that output is not written
            assert torch.equal(a, b), name


def test_calls_left_to_python(ops):
    n = ops._calls
    x = torch.randn(4, 32, device="cuda").to(torch.bfloat16)
    assert n.dynamic_quant(x, False) is not None
    wide = torch.randn(4, 64, device="cuda").to(torch.bfloat16)
    assert n.dynamic_quant(wide[:, ::2], False) is None  # strided
    assert n.dynamic_quant(x.cpu(), False) is None
    assert n.dynamic_quant(x.float(), False) is None
    assert n.dynamic_quant(x[:0], False) is None
    assert n.dynamic_quant(x[0], False) is None
    assert n.dynamic_quant("x", False) is None and n.dynamic_quant(x, 1) is None

    class Sub(torch.Tensor):
        pass

    assert n.dynamic_quant(x.as_subclass(Sub), False) is None
    with torch.overrides.BaseTorchFunctionMode():
        assert n.dynamic_quant(x, False) is None
    i8 = torch.ones((4, 24), dtype=torch.int8, device="cuda")
    w = torch.ones((24, 48), dtype=torch.int8, device="cuda")
    scale = torch.ones((48,), device="cuda")
    assert n.quant_matmul(i8, w, scale, None, None, None, None, False) is None  # K no multiple of 16: refused by the library
    with pytest.raises(RuntimeError):
        ops.quant_matmul(i8, w, scale)
    for bad in ([1, 2], [3, 2, 4], [-1, 2, 4], [1, 2, 3], [1.0, 2, 4]):
        assert n.grouped_matmul(x, torch.zeros((3, 32, 16), dtype=torch.bfloat16, device="cuda"), bad, None, False, None,
                                None) is None
