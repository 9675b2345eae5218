"""The work this framework is used for on one GPU, case by case, through its public entry points.

Five kinds of work, each over the range it is used in:

  mlp       ``TensorParallelMLP.forward``: the gated MLP block of a Llama-3-70B-like layer (hidden 8192, intermediate 28672, or the
            share of one rank at a tensor-parallel degree of 4 or 8), from one decoded token to an 8192-token prefill
  gemm      ``ops.gemm.gemm`` / ``gemm_swiglu`` on their own, both epilogues, sizes that are no multiple of a tile
  moe       ``ExpertParallelMoE.forward``: router, dispatch, experts, combine (hidden 7168, 32 experts of 2048 on this GPU, top-8:
            what one of eight GPUs holds of 256 experts), decode and prefill
  exchange  ``ExpertParallelContext``: route, dispatch and combine around experts that cost one pass over their rows
  emulated  the collectives, as ``world`` virtual ranks on one GPU (``EmulatedWorld``): latency packets, staged and chunked
            bands, copies and reductions, bf16 / fp16 / fp32
"""
import math

import torch

AR, AG, RS, A2A = 0, 1, 3, 5                                    # purlin_b200.Collective
COLLECTIVES = {"all_reduce": AR, "all_gather": AG, "reduce_scatter": RS, "all_to_all": A2A}
DTYPES = {"bf16": (0, torch.bfloat16), "fp16": (1, torch.float16), "fp32": (4, torch.float32)}


def listed():
    return [
        # one decoded token on the weights of one rank at TP = 8: bound by reading the weights
        {"name": "mlp_decode_1", "kind": "mlp", "tokens": 1, "hidden": 8192, "intermediate": 3584},
        # a decode batch on the whole block
        {"name": "mlp_decode_64", "kind": "mlp", "tokens": 64, "hidden": 8192, "intermediate": 28672},
        # a chunk of a prompt that is no multiple of any tile, TP = 4 share
        {"name": "mlp_chunk_1000", "kind": "mlp", "tokens": 1000, "hidden": 8192, "intermediate": 7168},
        # a full prefill: the workload of bench.py
        {"name": "mlp_prefill_8192", "kind": "mlp", "tokens": 8192, "hidden": 8192, "intermediate": 28672},
        # the smallest GEMM of the tests: one launch, remainders in every dimension
        {"name": "gemm_200x264x72", "kind": "gemm", "m": 200, "n": 264, "k": 72, "swiglu": False},
        # MoE layer of one of eight GPUs: a decode batch (each expert sees a few dozen rows) and a prefill
        {"name": "moe_decode_128", "kind": "moe", "tokens": 128, "hidden": 7168, "intermediate": 2048, "experts": 32, "topk": 8},
        {"name": "moe_prefill_4096", "kind": "moe", "tokens": 4096, "hidden": 7168, "intermediate": 2048, "experts": 32, "topk": 8},
        # the token exchange by itself: an odd decode batch on small rows, and the MoE benchmark's shape
        {"name": "exchange_300", "kind": "exchange", "tokens": 300, "hidden": 1024, "experts": 64, "topk": 8},
        {"name": "exchange_4096", "kind": "exchange", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8},
        # collectives: a decode-sized all-reduce (packets), an activation-sized reduce-scatter in fp32 with an odd size, a
        # gradient-bucket-sized all-reduce
        {"name": "all_reduce_8k_w8", "kind": "emulated", "collective": "all_reduce", "world": 8, "bytes": 8192, "dtype": "bf16"},
        {"name": "reduce_scatter_odd_w2", "kind": "emulated", "collective": "reduce_scatter", "world": 2, "bytes": 1000032, "dtype": "fp32"},
        {"name": "all_reduce_64m_w4", "kind": "emulated", "collective": "all_reduce", "world": 4, "bytes": 64 << 20, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "mlp", "gemm", "moe", "exchange", "emulated"])
    if kind == "mlp":
        return {"kind": kind, "tokens": _log(rng, 1, 8192), "hidden": 8 * _log(rng, 128, 1024), "intermediate": 16 * _log(rng, 64, 1792)}
    if kind == "gemm":
        swiglu = rng.random() < 0.3
        n = 32 * _log(rng, 2, 256) if swiglu else 8 * _log(rng, 8, 1024)
        return {"kind": kind, "m": _log(rng, 1, 8192), "n": n, "k": 8 * _log(rng, 8, 1024), "swiglu": swiglu}
    if kind == "moe":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "hidden": 64 * _log(rng, 16, 112), "intermediate": 64 * _log(rng, 4, 32),
                "experts": rng.choice([32, 64]), "topk": rng.choice([1, 2, 4, 6, 8])}
    if kind == "exchange":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "hidden": 16 * _log(rng, 32, 448), "experts": rng.choice([32, 64, 128, 256]),
                "topk": rng.choice([1, 2, 4, 6, 8])}
    name = rng.choice(sorted(COLLECTIVES))
    world = rng.choice([2, 4, 8])
    total = _log(rng, 4096, 64 << 20)                              # bytes of the larger of a rank's two buffers
    return {"kind": kind, "collective": name, "world": world, "bytes": max(32, (total if name == "all_reduce" else total // world) // 32 * 32),
            "dtype": rng.choice(sorted(DTYPES))}


# ------------------------------------------------------------------------------------------------------------------------
# inputs: activations N(0, 1), weights N(0, 0.02) as the framework's own models initialise them
# ------------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _mlp_inputs(c, seed):
    g = _gen(seed)
    gate = _randn(g, c["intermediate"], c["hidden"], scale=0.02)
    up = _randn(g, c["intermediate"], c["hidden"], scale=0.02)
    down = _randn(g, c["hidden"], c["intermediate"], scale=0.02)
    return gate, up, down, _randn(g, c["tokens"], c["hidden"])


def _gemm_inputs(c, seed):
    g = _gen(seed)
    a = _randn(g, c["m"], c["k"])
    if c["swiglu"]:
        return a, (_randn(g, c["n"] // 2, c["k"], scale=0.05), _randn(g, c["n"] // 2, c["k"], scale=0.05))
    return a, (_randn(g, c["n"], c["k"], scale=0.05),)


def _moe_inputs(c, seed):
    g = _gen(seed)
    e, h, i = c["experts"], c["hidden"], c["intermediate"]
    router = _randn(g, e, h, scale=0.02)
    gate = torch.stack([_randn(g, i, h, scale=0.02) for _ in range(e)])
    up = torch.stack([_randn(g, i, h, scale=0.02) for _ in range(e)])
    down = torch.stack([_randn(g, h, i, scale=0.02) for _ in range(e)])
    return router, gate, up, down, _randn(g, c["tokens"], h)


def _exchange_inputs(c, seed):
    g = _gen(seed)
    return _randn(g, c["tokens"], c["experts"], dtype=torch.float32), _randn(g, c["tokens"], c["hidden"])


def _emulated_sizes(c):
    """(input bytes, output bytes) of one rank."""
    n, w = c["bytes"], c["world"]
    return {"all_reduce": (n, n), "all_gather": (n, n * w), "reduce_scatter": (n * w, n), "all_to_all": (n * w, n * w)}[c["collective"]]


def _emulated_inputs(c, seed):
    g = _gen(seed)
    dtype = DTYPES[c["dtype"]][1]
    return [_randn(g, _emulated_sizes(c)[0] // dtype.itemsize, dtype=dtype) for _ in range(c["world"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        from purlin_b200.models.tp_mlp import TensorParallelMLP
        from purlin_b200.ops.gemm import interleave_gate_up
        mlp = TensorParallelMLP(case["hidden"], case["intermediate"], case["tokens"], device="cuda:0")
        mlp.w_gate, mlp.w_up, mlp.w_down, x = _mlp_inputs(case, seed)     # as a checkpoint would be loaded
        mlp.w_gu = interleave_gate_up(mlp.w_gate, mlp.w_up)
        return {"kind": kind, "mlp": mlp, "x": x}
    if kind == "gemm":
        from purlin_b200.ops.gemm import interleave_gate_up
        a, w = _gemm_inputs(case, seed)
        return {"kind": kind, "a": a, "w": interleave_gate_up(*w) if case["swiglu"] else w[0], "swiglu": case["swiglu"]}
    if kind == "moe":
        from purlin_b200.models.moe_block import ExpertParallelMoE
        from purlin_b200.ops.gemm import interleave_gate_up
        moe = ExpertParallelMoE(case["hidden"], case["intermediate"], case["experts"], case["topk"], max_tokens=case["tokens"],
                                device="cuda:0", capacity_factor=1.0)
        moe.w_router, moe.w_gate, moe.w_up, moe.w_down, x = _moe_inputs(case, seed)
        moe.w_gu = torch.stack([interleave_gate_up(a, b) for a, b in zip(moe.w_gate, moe.w_up)])
        return {"kind": kind, "moe": moe, "x": x}
    if kind == "exchange":
        from purlin_b200.parallel.expert_parallel import ExpertParallelContext
        logits, x = _exchange_inputs(case, seed)
        ep = ExpertParallelContext(None, "cuda:0", max_tokens=case["tokens"], hidden=case["hidden"], experts=case["experts"],
                                   topk=case["topk"], capacity_factor=1.0)
        return {"kind": kind, "ep": ep, "logits": logits, "x": x, "rows": case["tokens"] * case["topk"]}
    from purlin_b200.utils.emulation import EmulatedWorld
    ins = _emulated_inputs(case, seed)
    largest = max(_emulated_sizes(case))
    staging = min(max(1 << 20, (largest + 31) // 32 * 32), 256 << 20)     # every rank's whole buffer fits
    outs = [torch.empty(_emulated_sizes(case)[1] // t.element_size(), dtype=t.dtype, device="cuda") for t in ins]
    return {"kind": kind, "world": EmulatedWorld(case["world"], staging), "ins": ins, "outs": outs,
            "collective": COLLECTIVES[case["collective"]], "bytes": case["bytes"], "dtype": DTYPES[case["dtype"]][0]}


def run(state):
    kind = state["kind"]
    if kind == "mlp":
        return state["mlp"].forward(state["x"])
    if kind == "gemm":
        from purlin_b200.ops.gemm import gemm, gemm_swiglu
        return (gemm_swiglu if state["swiglu"] else gemm)(state["a"], state["w"])
    if kind == "moe":
        return state["moe"].forward(state["x"])
    if kind == "exchange":
        ep, x = state["ep"], state["x"]
        experts, weights = ep.route(state["logits"], normalize=False)
        rows, counts = ep.dispatch(x)
        torch.mul(rows[: state["rows"]], 0.5, out=ep.out_rows()[: state["rows"]])      # the experts
        return {"experts": experts, "weights": weights, "counts": counts, "y": ep.combine(x.shape[0])}
    state["world"].run(state["collective"], state["ins"], state["outs"], nbytes=state["bytes"], dtype=state["dtype"])
    return state["outs"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "mlp":
        t, h, i = c["tokens"], c["hidden"], c["intermediate"]
        return {"bytes": 6 * h * i + 4 * t * h, "flops": 6 * t * h * i}
    if kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * (m * k + n * k + m * (n // 2 if c["swiglu"] else n)), "flops": 2 * m * n * k}
    if kind == "moe":
        t, h, i, e, k = c["tokens"], c["hidden"], c["intermediate"], c["experts"], c["topk"]
        used = e * (1 - (1 - k / e) ** t)                          # experts that any token chose, on average
        return {"bytes": used * 6 * h * i + 2 * e * h + 4 * t * h, "flops": 6 * t * k * h * i + 2 * t * e * h}
    if kind == "exchange":
        t, h, e, k = c["tokens"], c["hidden"], c["experts"], c["topk"]
        return {"bytes": 4 * t * e + 8 * t * k + 2 * t * h * (2 + 4 * k), "flops": 3 * t * k * h}
    w, (a, b) = c["world"], _emulated_sizes(c)
    adds = w * b / DTYPES[c["dtype"]][1].itemsize * (w - 1) if c["collective"] in ("all_reduce", "reduce_scatter") else 0
    return {"bytes": w * (a + b), "flops": adds}


def tolerance(case):
    kind = case["kind"]
    if kind == "mlp":
        return {"rel": 1e-2}                                       # bf16 products and a bf16 intermediate: 2.4e-3 against 64 bits
    if kind == "gemm":
        return {"rel": 1e-2 if case["swiglu"] else 7e-3}           # one rounding to bf16: 1.7e-3 against 64 bits
    if kind == "moe":
        return {"rel": 1.2e-2, "max": 0.9}                         # 2.9e-3; bf16 logits: a token near a tie may choose another expert
    if kind == "exchange":
        return {"rel": 7e-3, "differ": 1e-3}
    if case["collective"] in ("all_gather", "all_to_all"):
        return "exact"
    return {"rel": {"bf16": 7e-3, "fp16": 1e-3, "fp32": 1e-6}[case["dtype"]]}


def exact(case, seed):
    kind = case["kind"]
    silu = torch.nn.functional.silu
    if kind == "mlp":
        gate, up, down, x = _mlp_inputs(case, seed)
        x = x.double()
        h = silu(x @ gate.double().t())
        h *= x @ up.double().t()
        return h @ down.double().t()
    if kind == "gemm":
        a, w = _gemm_inputs(case, seed)
        p = [a.double() @ v.double().t() for v in w]
        return silu(p[0]) * p[1] if case["swiglu"] else p[0]
    if kind == "moe":
        router, gate, up, down, x = _moe_inputs(case, seed)
        x = x.double()
        probs = torch.softmax((x @ router.double().t()).to(torch.bfloat16).double(), -1)      # the router's logits are bf16 by definition
        order = torch.sort(probs, dim=-1, descending=True, stable=True)
        w, idx = order.values[:, : case["topk"]], order.indices[:, : case["topk"]]
        w = w / w.sum(-1, keepdim=True)
        y = torch.zeros_like(x)
        for e in range(case["experts"]):
            tok, k = (idx == e).nonzero(as_tuple=True)
            if tok.numel():
                xe = x[tok]
                h = silu(xe @ gate[e].double().t()) * (xe @ up[e].double().t())
                y.index_add_(0, tok, (h @ down[e].double().t()) * w[tok, k].unsqueeze(-1))
        return y
    if kind == "exchange":
        logits, x = _exchange_inputs(case, seed)
        weights = torch.sort(torch.softmax(logits.double(), -1), dim=-1, descending=True, stable=True).values[:, : case["topk"]]
        return {"experts": None, "weights": weights, "counts": None, "y": 0.5 * x.double() * weights.sum(-1, keepdim=True)}
    ins, w = [t.double() for t in _emulated_inputs(case, seed)], case["world"]
    if case["collective"] == "all_reduce":
        return [sum(ins)] * w
    if case["collective"] == "all_gather":
        return [torch.cat(ins)] * w
    if case["collective"] == "reduce_scatter":
        return list(sum(ins).chunk(w))
    return [torch.cat([t.chunk(w)[r] for t in ins]) for r in range(w)]
