"""Per-channel vectors that start inside a larger tensor: at 16 bytes they are taken, with the same bits; elsewhere the call
is refused on the host, by the operator functions (both halves) and the registered operators; single values may lie
anywhere."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _moved(t, off):
    """`t` as a contiguous view that starts `off` elements into its storage."""
    held = torch.empty((t.numel() + off,), dtype=t.dtype, device=t.device)
    held[off:].copy_(t.reshape(-1))
    return held[off:].view(t.shape)


def _dense(ops, **moved):
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randint(-127, 128, (40, 64), generator=g, device="cuda", dtype=torch.int8)
    w = torch.randint(-127, 128, (64, 48), generator=g, device="cuda", dtype=torch.int8)
    vec = {"scale": torch.rand((48,), generator=g, device="cuda"), "offset": torch.rand((48,), generator=g, device="cuda"),
           "bias": torch.rand((48,), generator=g, device="cuda").bfloat16()}
    vec = {k: _moved(v, moved[k]) if k in moved else v for k, v in vec.items()}
    return ops.quant_matmul(x, w, vec["scale"], offset=vec["offset"], bias=vec["bias"])


@pytest.fixture(params=["native", "python", "plugin"])
def route(request, ops, monkeypatch):
    if request.param == "plugin":
        import cannbench_operator_solutions_b200 as pkg

        pkg.load_torch_plugin()
        return torch.ops.cann_bench
    if request.param == "python":
        monkeypatch.setattr(ops, "_calls", None)
    return ops


@pytest.mark.parametrize("name,taken,refused", [("scale", (4, 12), (1, 2)), ("offset", (8,), (3,)), ("bias", (8, 16), (1, 4))])
def test_dense(route, name, taken, refused):
    want = _dense(route)
    for off in taken:
        assert torch.equal(_dense(route, **{name: off}), want)
    for off in refused:
        with pytest.raises(RuntimeError, match="align"):
            _dense(route, **{name: off})


def test_single_values(route):
    x = torch.ones((5, 32), dtype=torch.int8, device="cuda")
    w = torch.ones((32, 16), dtype=torch.int8, device="cuda")
    for dtype in (torch.float32, torch.bfloat16):
        got = route.quant_matmul(x, w, _moved(torch.full((1,), 0.5, device="cuda", dtype=dtype), 3),
                                 offset=_moved(torch.ones((1,), device="cuda"), 1),
                                 bias=_moved(torch.full((1,), 2.0, device="cuda", dtype=dtype), 1))
        assert (got == 19.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_grouped_bias(route, dtype):
    x = torch.ones((5, 32), dtype=dtype, device="cuda")
    w = torch.ones((2, 32, 16), dtype=dtype, device="cuda")
    bias = torch.arange(32, device="cuda").to(dtype).view(2, 16)
    want = route.grouped_matmul(x, w, [2, 5], bias, 2)[0]
    assert torch.equal(want, torch.cat([bias[:1].expand(2, 16), bias[1:].expand(3, 16)]) + 32)
    assert torch.equal(route.grouped_matmul(x, w, [2, 5], _moved(bias, 8), 2)[0], want)
    with pytest.raises(RuntimeError, match="align"):
        route.grouped_matmul(x, w, [2, 5], _moved(bias, 1), 2)


def test_grouped_scale(route):
    x = torch.ones((5, 32), dtype=torch.int8, device="cuda")
    w = torch.ones((2, 32, 16), dtype=torch.int8, device="cuda")
    xs, ws = _moved(torch.ones((5,), device="cuda"), 1), torch.full((2, 16), 0.5, device="cuda")

    def call(scale):
        if route is torch.ops.cann_bench:
            return route.grouped_matmul(x, w, [2, 5], None, 2, False, xs, scale)[0]
        return route.grouped_matmul(x, w, [2, 5], None, 2, False, x_scale=xs, weight_scale=scale)[0]

    assert (call(_moved(ws, 4)) == 16.0).all()
    with pytest.raises(RuntimeError, match="align"):
        call(_moved(ws, 3))
