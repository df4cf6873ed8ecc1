"""The work that users of this framework have it do, as timed cases.

Every case goes through the public entry points (the package's operator functions, the torch operators they mirror, and
the expert-parallel layer) on inputs of the distributions the W8A8 path meets: N(0,1) activations, uniform int8
weights with per-channel scales, softmax routing or Zipf-skewed expert loads.

Kinds:
  linear    dynamic_quant -> quant_matmul through torch.ops.cann_bench: one quantised linear layer
  ffn       add_rms_norm_dynamic_quant -> quant_matmul -> dequant_swiglu_quant -> quant_matmul: one dense layer
  norm      add_rms_norm_dynamic_quant alone
  router    moe_gating_top_k_softmax on the router's logits
  up        grouped_matmul_swiglu_quant alone (up projection of all experts)
  moe       the expert layer as a step: normalise, route, dispatch, both grouped matmuls, combine
  grouped   grouped_matmul on 16-bit or fp32 operands (the reference's float path)
  exchange  moe_re_routing of received int8 rows, moe_finalize_routing of the experts' outputs
  swiglu    dequant_swiglu_quant of an int32 matmul result
"""
import math

import torch

import cannbench_operator_solutions_b200 as w8a8
from cannbench_operator_solutions_b200 import ep

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # the smallest call: one quantised linear layer on a short batch
        {"name": "linear_small", "kind": "linear", "rows": 128, "k": 1024, "n": 1024, "dtype": "bf16", "bias": False},
        # prefill of a long batch through the largest dense projection
        {"name": "linear_prefill", "kind": "linear", "rows": 8192, "k": 7168, "n": 18432, "dtype": "bf16", "bias": False},
        # a dense layer in decode: few rows, bound by reading both weight matrices
        {"name": "ffn_decode", "kind": "ffn", "rows": 16, "hidden": 7168, "inter": 9216, "dtype": "bf16", "bias": False},
        # the same layer in prefill of a ragged batch, fp16, with bias
        {"name": "ffn_prefill_ragged", "kind": "ffn", "rows": 1531, "hidden": 7168, "inter": 9216, "dtype": "fp16", "bias": True},
        # residual add + normalisation + quantisation of a prefill batch
        {"name": "norm_prefill", "kind": "norm", "rows": 8192, "hidden": 7168, "dtype": "bf16"},
        # router of the largest batch
        {"name": "router_prefill", "kind": "router", "rows": 65536, "experts": 256, "topk": 8, "dtype": "bf16"},
        # up projection of 256 experts under a Zipf-skewed load
        {"name": "up_zipf", "kind": "up", "rows": 131072, "experts": 256, "hidden": 7168, "inter": 2048, "skew": 1.1},
        # expert layer in decode: every expert sees a few rows at most
        {"name": "moe_decode", "kind": "moe", "rows": 64, "experts": 256, "topk": 8, "hidden": 7168, "inter": 2048, "dtype": "bf16"},
        # expert layer, the largest batch
        {"name": "moe_prefill", "kind": "moe", "rows": 65536, "experts": 256, "topk": 8, "hidden": 7168, "inter": 2048, "dtype": "bf16"},
        # down projection of experts kept in bf16, ragged group sizes
        {"name": "grouped_bf16", "kind": "grouped", "rows": 8000, "experts": 32, "k": 2048, "n": 7168, "dtype": "bf16", "bias": True},
        # rows of 8 ranks regrouped by expert, then the experts' rows combined per token
        {"name": "exchange_prefill", "kind": "exchange", "rows": 65536, "ranks": 8, "experts": 32, "topk": 8, "hidden": 7168, "dtype": "bf16"},
        # activation of an int32 up projection with smooth scales
        {"name": "swiglu_int32", "kind": "swiglu", "rows": 16384, "inter": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log16(rng, lo, hi):
    return max(lo, min(hi, int(round(_log(rng, lo, hi) / 16.0)) * 16))


def draw(rng):
    kind = rng.choice(["linear", "ffn", "norm", "router", "up", "moe", "grouped", "exchange", "swiglu"])
    half = rng.choice(["bf16", "fp16"])
    if kind == "linear":
        return {"kind": kind, "rows": _log(rng, 1, 8192), "k": _log16(rng, 512, 7168), "n": _log16(rng, 512, 18432),
                "dtype": half, "bias": rng.random() < 0.5}
    if kind == "ffn":
        return {"kind": kind, "rows": _log(rng, 1, 4096), "hidden": _log16(rng, 1024, 7168),
                "inter": _log16(rng, 1024, 9216), "dtype": half, "bias": rng.random() < 0.5}
    if kind == "norm":
        return {"kind": kind, "rows": _log(rng, 1, 16384), "hidden": _log16(rng, 1024, 8192), "dtype": half}
    if kind == "router":
        experts = rng.choice([32, 60, 64, 128, 160, 256])
        return {"kind": kind, "rows": _log(rng, 16, 65536), "experts": experts, "topk": rng.choice([1, 2, 4, 6, 8]),
                "dtype": rng.choice(["bf16", "fp16", "fp32"])}
    if kind == "up":
        return {"kind": kind, "rows": _log(rng, 64, 65536), "experts": rng.choice([8, 32, 64, 128]),
                "hidden": _log16(rng, 1024, 7168), "inter": _log16(rng, 512, 2048), "skew": round(rng.uniform(0.0, 1.2), 2)}
    if kind == "moe":
        return {"kind": kind, "rows": _log(rng, 1, 16384), "experts": rng.choice([16, 32, 64, 128]),
                "topk": rng.choice([2, 4, 8]), "hidden": _log16(rng, 1024, 7168), "inter": _log16(rng, 512, 2048),
                "dtype": half}
    if kind == "grouped":
        return {"kind": kind, "rows": _log(rng, 64, 16384), "experts": rng.choice([4, 8, 16, 32]),
                "k": _log16(rng, 512, 4096), "n": _log16(rng, 512, 7168),
                "dtype": rng.choice(["bf16", "fp16", "fp32"]), "bias": rng.random() < 0.5}
    if kind == "exchange":
        return {"kind": kind, "rows": _log(rng, 64, 65536), "ranks": rng.choice([2, 4, 8]),
                "experts": rng.choice([8, 16, 32]), "topk": rng.choice([2, 4, 8]), "hidden": _log16(rng, 1024, 7168),
                "dtype": half}
    return {"kind": kind, "rows": _log(rng, 16, 16384), "inter": _log16(rng, 512, 4096)}


# ---------------------------------------------------------------------------------------------- inputs
class _Gen:
    """Seeded inputs on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, generator=self.g, device="cuda") * (hi - lo) + lo

    def int8(self, *shape):
        return torch.randint(-127, 128, shape, generator=self.g, device="cuda", dtype=torch.int8)

    def channel_scale(self, depth, *shape):
        """Weight scales that keep an output of `depth` unit-variance terms near unit variance."""
        return self.uniform(0.5, 1.5, *shape) / (73.0 * math.sqrt(depth))

    def gamma(self, n, dtype):
        return (1.0 + 0.1 * self.normal(n)).to(dtype)

    def group_ends(self, rows, experts, skew):
        """Cumulative group list of `rows` rows spread over the experts with Zipf weights (skew 0: even odds)."""
        w = torch.arange(1, experts + 1, device="cuda", dtype=torch.float64).pow(-skew)
        w = w[torch.randperm(experts, generator=self.g, device="cuda")]
        pick = torch.multinomial(w.float(), rows, replacement=True, generator=self.g)
        return torch.bincount(pick, minlength=experts).cumsum(0)


def prepare(case, seed):
    g = _Gen(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "linear":
        w8a8.load_torch_plugin()
        dt, k, n = _DTYPES[case["dtype"]], case["k"], case["n"]
        s.update(x=g.normal(case["rows"], k, dtype=dt), w=g.int8(k, n), scale=g.channel_scale(k, n),
                 bias=(0.02 * g.normal(n)).to(dt) if case["bias"] else None,
                 out="bfloat16" if case["dtype"] == "bf16" else "float16")
    elif kind == "ffn":
        dt, h, i = _DTYPES[case["dtype"]], case["hidden"], case["inter"]
        s.update(x=g.normal(case["rows"], h, dtype=dt), residual=g.normal(case["rows"], h, dtype=dt),
                 gamma=g.gamma(h, dt), w_up=g.int8(h, 2 * i), s_up=g.channel_scale(h, 2 * i), w_down=g.int8(i, h),
                 s_down=g.channel_scale(i, h), b_up=None, b_down=None,
                 out="bfloat16" if case["dtype"] == "bf16" else "float16")
        if case["bias"]:
            s.update(b_up=(0.02 * g.normal(2 * i)).to(dt), b_down=(0.02 * g.normal(h)).to(dt))
    elif kind == "norm":
        dt, h = _DTYPES[case["dtype"]], case["hidden"]
        s.update(x=g.normal(case["rows"], h, dtype=dt), residual=g.normal(case["rows"], h, dtype=dt), gamma=g.gamma(h, dt))
    elif kind == "router":
        s.update(x=g.normal(case["rows"], case["experts"]).to(_DTYPES[case["dtype"]]), topk=case["topk"])
    elif kind == "up":
        m, e, h, i = case["rows"], case["experts"], case["hidden"], case["inter"]
        s.update(x=g.int8(m, h), x_scale=g.uniform(1e-3, 5e-2, m), w=g.int8(e, h, 2 * i),
                 s_up=g.channel_scale(h, e, 2 * i), ends=g.group_ends(m, e, case["skew"]).tolist())
    elif kind == "moe":
        dt, m, e, h, i = _DTYPES[case["dtype"]], case["rows"], case["experts"], case["hidden"], case["inter"]
        shard = ep.ExpertShard(g.int8(e, h, 2 * i), g.channel_scale(h, e, 2 * i), g.int8(e, i, h),
                               g.channel_scale(i, e, h))
        probs, idx = torch.softmax(g.normal(m, e), -1).topk(case["topk"], -1)
        s.update(layer=ep.MoeFfnChain(e, shard, transport="p2p"), x=g.normal(m, h, dtype=dt),
                 residual=g.normal(m, h, dtype=dt), gamma=g.gamma(h, dt), idx=idx.to(torch.int32).contiguous(),
                 probs=(probs / probs.sum(-1, keepdim=True)).contiguous())
    elif kind == "grouped":
        dt, m, e, k, n = _DTYPES[case["dtype"]], case["rows"], case["experts"], case["k"], case["n"]
        s.update(x=g.normal(m, k, dtype=dt), w=g.normal(e, k, n, dtype=dt).mul_(1.0 / math.sqrt(k)),
                 bias=(0.02 * g.normal(e, n)).to(dt) if case["bias"] else None,
                 ends=g.group_ends(m, e, 0.5).tolist())
    elif kind == "exchange":
        dt, m, k, h = _DTYPES[case["dtype"]], case["rows"], case["topk"], case["hidden"]
        cells = case["ranks"] * case["experts"]
        counts = torch.bincount(torch.randint(0, cells, (m,), generator=g.g, device="cuda"), minlength=cells)
        tokens = max(1, m // k)
        s.update(x=g.int8(m, h), x_scale=g.uniform(1e-3, 5e-2, m), counts=counts.view(case["ranks"], case["experts"]),
                 rows=g.normal(tokens * k, h, dtype=dt),
                 pos=torch.randperm(tokens * k, generator=g.g, device="cuda").to(torch.int32),
                 skip=g.normal(tokens, h, dtype=dt), probs=torch.softmax(g.normal(tokens, k), -1))
    else:
        m, i = case["rows"], case["inter"]
        s.update(x=(g.normal(m, 2 * i) * 60000.0).to(torch.int32), w_scale=g.uniform(1e-3, 1e-2, 2 * i),
                 x_scale=g.uniform(1e-3, 1e-2, m), smooth=g.uniform(0.5, 2.0, i))
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "linear":
        q, qs = torch.ops.cann_bench.dynamic_quant(s["x"])
        return torch.ops.cann_bench.quant_matmul(q, s["w"], s["scale"], pertoken_scale=qs, bias=s["bias"],
                                                 output_dtype=s["out"])
    if kind == "ffn":
        q, residual, qs = w8a8.add_rms_norm_dynamic_quant(s["x"], s["residual"], s["gamma"], 1e-6)
        h = w8a8.quant_matmul(q, s["w_up"], s["s_up"], pertoken_scale=qs, bias=s["b_up"], output_dtype=s["out"])
        a, a_scale = w8a8.dequant_swiglu_quant(h, activate_left=True)
        out = w8a8.quant_matmul(a, s["w_down"], s["s_down"], pertoken_scale=a_scale, bias=s["b_down"],
                                output_dtype=s["out"])
        return out, residual
    if kind == "norm":
        return w8a8.add_rms_norm_dynamic_quant(s["x"], s["residual"], s["gamma"], 1e-6)
    if kind == "router":
        return w8a8.moe_gating_top_k_softmax(s["x"], None, s["topk"])
    if kind == "up":
        return w8a8.grouped_matmul_swiglu_quant(s["x"], s["w"], s["s_up"], s["x_scale"], s["ends"])
    if kind == "moe":
        return s["layer"].forward(s["x"], s["residual"], s["gamma"], 1e-6, s["idx"], s["probs"])
    if kind == "grouped":
        return w8a8.grouped_matmul(s["x"], s["w"], s["ends"], s["bias"], 3)
    if kind == "exchange":
        regrouped = w8a8.moe_re_routing(s["x"], s["counts"], s["x_scale"])
        combined = w8a8.moe_finalize_routing(s["rows"], s["pos"], s["skip"], None, None, s["probs"], None, 0)
        return regrouped, combined
    return w8a8.dequant_swiglu_quant(s["x"], s["w_scale"], s["x_scale"], s["smooth"], True)


# ------------------------------------------------------------------------------------------------ what it needs
def _touched(case):
    """Experts that at least one row is routed to, as expected from even odds."""
    pairs = case["rows"] * case["topk"]
    return case["experts"] * (1.0 - (1.0 - 1.0 / case["experts"]) ** pairs)


def work(case):
    kind, m = case["kind"], case["rows"]
    if kind == "linear":
        k, n = case["k"], case["n"]
        return {"bytes": 2 * m * k + k * n + 4 * n + 2 * m * n, "flops": 2.0 * m * k * n}
    if kind == "ffn":
        h, i = case["hidden"], case["inter"]
        return {"bytes": 3 * h * i + 4 * (2 * i + h) + 8 * m * h + 2 * h, "flops": 6.0 * m * h * i}
    if kind == "norm":
        return {"bytes": m * (7 * case["hidden"] + 4) + 2 * case["hidden"], "flops": 6.0 * m * case["hidden"]}
    if kind == "router":
        size = 4 if case["dtype"] == "fp32" else 2
        return {"bytes": m * (case["experts"] * size + case["topk"] * (size + 8)), "flops": 10.0 * m * case["experts"]}
    if kind == "up":
        h, i, e = case["hidden"], case["inter"], case["experts"]
        return {"bytes": e * (2 * h * i + 8 * i) + m * (h + 4) + m * (i + 4), "flops": 4.0 * m * h * i}
    if kind == "moe":
        h, i, k = case["hidden"], case["inter"], case["topk"]
        return {"bytes": _touched(case) * (3 * h * i + 4 * (2 * i + h)) + 8 * m * h + 8 * m * k, "flops": 6.0 * m * k * h * i}
    if kind == "grouped":
        size, k, n = 4 if case["dtype"] == "fp32" else 2, case["k"], case["n"]
        return {"bytes": size * (m * k + case["experts"] * k * n + m * n), "flops": 2.0 * m * k * n}
    if kind == "exchange":
        h, k = case["hidden"], case["topk"]
        tokens = max(1, m // k)
        return {"bytes": m * (2 * h + 12) + tokens * (2 * k * h + 4 * h + 8 * k), "flops": 2.0 * tokens * k * h}
    return {"bytes": m * (9 * case["inter"] + 8) + 12 * case["inter"], "flops": 10.0 * m * case["inter"]}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _narrow64(v):
    """fp32 -> fp16 -> int8 of the operators, ties to even both times, on values held in 64 bits."""
    return v.to(torch.float16).double().round().clamp_(-128.0, 127.0)


def _quant64(v):
    amax = v.abs().amax(-1, keepdim=True).clamp_min(1e-12)
    return _narrow64(v * (127.0 / amax)), (amax / 127.0).squeeze(-1)


def _norm64(s):
    """(int8 values, residual sum, per-row scale) of add_rms_norm_dynamic_quant."""
    total = s["x"].double() + s["residual"].double()
    z = total * s["gamma"].double()
    rstd = (total.square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    q, scale = _quant64(z * rstd)
    return q, total, scale


def _matmul64(q, q_scale, w, w_scale, bias=None):
    out = (q @ w.double()) * w_scale.double() * q_scale.unsqueeze(-1)
    return out if bias is None else out + bias.double()


def _swiglu64(gate, up):
    return gate * torch.sigmoid(gate) * up


def exact(case, seed):
    """The floating results of `run` on the same inputs, worked out by torch in 64 bits; None beside int8 and index outputs."""
    s = prepare(case, seed)
    kind = s["kind"]
    if kind == "linear":
        q, qs = _quant64(s["x"].double())
        return _matmul64(q, qs, s["w"], s["scale"], s["bias"])
    if kind == "ffn":
        q, total, qs = _norm64(s)
        h = _matmul64(q, qs, s["w_up"], s["s_up"], s["b_up"]).to(s["x"].dtype).double()
        gate, up = h.chunk(2, -1)
        a, a_scale = _quant64(_swiglu64(gate, up))
        return _matmul64(a, a_scale, s["w_down"], s["s_down"], s["b_down"]), total
    if kind == "norm":
        _, total, scale = _norm64(s)
        return None, total, scale
    if kind == "router":
        return torch.softmax(s["x"].double(), -1).topk(s["topk"], -1).values, None, None
    if kind == "up":
        scale = torch.empty(case["rows"], dtype=torch.float64, device="cuda")
        first = 0
        for e, end in enumerate(s["ends"]):
            h = _matmul64(s["x"][first:end].double(), s["x_scale"][first:end].double(), s["w"][e], s["s_up"][e])
            gate, up = h.chunk(2, -1)
            scale[first:end] = _quant64(_swiglu64(gate, up))[1]
            first = end
        return None, scale
    if kind == "moe":
        q, total, qs = _norm64(s)
        shard, out = s["layer"].shard, torch.zeros_like(total)
        for e in range(case["experts"]):
            token, slot = torch.nonzero(s["idx"] == e, as_tuple=True)
            if token.numel() == 0:
                continue
            gate, up = _matmul64(q[token], qs[token], shard.w_up[e], shard.s_up[e]).chunk(2, -1)
            a, a_scale = _quant64(_swiglu64(gate, up))
            y = _matmul64(a, a_scale, shard.w_down[e], shard.s_down[e])
            out.index_add_(0, token, y * s["probs"][token, slot].double().unsqueeze(-1))
        return out, total
    if kind == "grouped":
        out = torch.empty(case["rows"], case["n"], dtype=torch.float64, device="cuda")
        first = 0
        for e, end in enumerate(s["ends"]):
            out[first:end] = s["x"][first:end].double() @ s["w"][e].double()
            if s["bias"] is not None:
                out[first:end] += s["bias"][e].double()
            first = end
        return [out]
    if kind == "exchange":
        cells = s["counts"].numel()
        cell = torch.repeat_interleave(torch.arange(cells, device="cuda"), s["counts"].flatten())
        order = torch.argsort(cell % case["experts"], stable=True)
        tokens, k = s["probs"].shape
        combined = s["skip"].double()
        for j in range(k):
            combined += s["rows"][s["pos"].view(k, tokens)[j].long()].double() * s["probs"][:, j:j + 1].double()
        return (None, s["x_scale"][order].double(), None, None), combined
    h = s["x"].double() * s["w_scale"].double() * s["x_scale"].double().unsqueeze(-1)
    gate, up = h.chunk(2, -1)
    return None, _quant64(_swiglu64(gate, up * s["smooth"].double()))[1]


# About four times what the path's results differ by from the same operation sequence carried out in 64 bits (2-norm,
# largest, and share of int8 values or indices that change), taken at reduced sizes of every kind.
_FP32_RESULTS = {"rel": 4e-7, "max": 1.5e-6, "differ": 5e-6}  # fp32 scales / probabilities beside int8 values or indices
_HALF_RESULTS = {"rel": 4e-4, "max": 3.6e-2}                  # one rounding step of bf16 / fp16 on a few elements
_FP32_PRODUCTS = {"rel": 8.5e-6, "max": 3.5e-5}               # fp32 sums of fp32 products


def tolerance(case):
    if case["kind"] in ("norm", "router", "up", "swiglu"):
        return dict(_FP32_RESULTS)
    if case["kind"] == "grouped" and case["dtype"] == "fp32":
        return dict(_FP32_PRODUCTS)
    return dict(_HALF_RESULTS)
