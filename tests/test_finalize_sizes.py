"""moe_finalize_routing refuses operands with fewer elements than its kernel reads, on the host and by every route."""
import pytest
import torch

SHORT = [("skip1", (6, 32)), ("skip2", (7, 31)), ("skip1", (32,)), ("scales", (6, 2)), ("expert_for_source_row", (13,)),
         ("expert_for_source_row", (1, 2))]


def _call(finalize, device, short=None, shape=None):
    shapes = {"skip1": (7, 32), "skip2": (7, 32), "bias": (3, 32), "scales": (7, 2), "expert_for_source_row": (7, 2)}
    if short is not None:
        shapes[short] = shape
    kw = {k: torch.ones(v, dtype=torch.int32 if k.startswith("expert") else torch.bfloat16, device=device)
          for k, v in shapes.items()}
    return finalize(torch.ones((14, 32), dtype=torch.bfloat16, device=device), torch.arange(14, dtype=torch.int32, device=device),
                    drop_pad_mode=2, **kw)


@pytest.mark.parametrize("short,shape", SHORT)
def test_operator_function_on_the_host(short, shape):
    from cannbench_operator_solutions_b200 import ops

    with pytest.raises(RuntimeError, match=f"{short} has too few elements"):
        _call(ops.moe_finalize_routing, "cpu", short, shape)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        _call(ops.moe_finalize_routing, "cpu")


@pytest.mark.gpu
@pytest.mark.parametrize("route", ["native", "python", "plugin"])
def test_every_route(ops, monkeypatch, route):
    if route == "plugin":
        import cannbench_operator_solutions_b200 as pkg

        pkg.load_torch_plugin()
        finalize = torch.ops.cann_bench.moe_finalize_routing
    else:
        finalize = ops.moe_finalize_routing
        if route == "python":
            monkeypatch.setattr(ops, "_calls", None)
    # 1 + 1 + (1 + 1) + (1 + 1); more elements than are read are as good
    assert (_call(finalize, "cuda") == 6.0).all()
    assert (_call(finalize, "cuda", "skip1", (9, 32)) == 6.0).all()
    for short, shape in SHORT:
        with pytest.raises(RuntimeError, match=f"{short} has too few elements"):
            _call(finalize, "cuda", short, shape)
