"""The work a user of this library has it do, as cases that can be timed and compared: plain projections, fused
projection + reduction layers, reductions of given partials, NVFP4 routed experts, and a whole block in the device loop.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges, `prepare(case, seed)` builds what a program
holds before the call (weights laid out, groups, captured graphs, inputs), `run(state)` is one pass through the public
entry points, `work(case)` what the pass cannot do without, and `tolerance(case)` how far another correct implementation
may be off. Everything runs on one GPU (a world-1 group), where a denoise round's row-parallel path is the same calls as
on several.

Two ways of calling are measured, the two a program has: `call` "graph" replays a captured CUDA graph (how an engine runs
its rounds) and "eager" makes the Python calls every time (warm-up, prefill, and programs that capture nothing).
"""

import math
from types import SimpleNamespace

import torch

from dlmrt_b200.distributed.parallel import Group
from dlmrt_b200.layers.linear import Linear
from dlmrt_b200.ops.block_graph import BlockGraph
from dlmrt_b200.quantization import nvfp4

DEVICE = "cuda:0"
EPS = 1e-6


def listed():
    return [
        # The smallest call: a shared expert's down-projection of a 32-token block, made from Python. Latency only.
        dict(name="linear_small", kind="linear", rows=32, n=2048, k=512, nn=False),
        # The largest: the self-conditioning soft embedding, softmax over the whole vocabulary times the tied embedding.
        dict(name="linear_vocab", kind="linear", rows=256, n=2560, k=151936, nn=True),
        # Eight layers of a dense 4B model's denoise round: o_proj and down_proj of a 256-token block, each fused with
        # residual + RMSNorm, in a graph. The benchmark's own layer shape.
        dict(name="dense_block256", kind="dense", rows=256, hidden=2560, k_o=4096, k_d=9728, layers=8, call="graph"),
        # The same pair at the width and block of a small MoE model (o_proj and shared-expert down-projection), 32 tokens:
        # weights are small and the launch chain counts.
        dict(name="dense_block32", kind="dense", rows=32, hidden=2048, k_o=2048, k_d=512, layers=20, call="graph"),
        # One layer called from Python with nothing round: 80 tokens, K that is no multiple of a k-block.
        dict(name="dense_odd", kind="dense", rows=80, hidden=2304, k_o=1000, k_d=4360, layers=1, call="eager"),
        # Reductions of partials that some other kernel produced: residual + norm, then a plain sum. A small block from
        # Python, and the widest hidden size with a full block in a graph.
        dict(name="reduce_small", kind="reduce", rows=32, hidden=2048, pairs=1, call="eager"),
        dict(name="reduce_wide", kind="reduce", rows=256, hidden=8192, pairs=8, call="graph"),
        # Four MoE layers of a 32-token block, 256 experts top-8, BF16 input, shared expert folded in, down-projection
        # fused with the reduction; routing spread evenly, and skewed (Zipf) as trained routers are.
        dict(name="moe_uniform", kind="moe", rows=32, hidden=2048, f=512, experts=256, top_k=8, layers=4, routing="uniform",
             activation="swiglu", shared=True, router=False, fused=True, call="graph"),
        dict(name="moe_zipf", kind="moe", rows=32, hidden=2048, f=512, experts=256, top_k=8, layers=4, routing="zipf",
             activation="swiglu", shared=True, router=False, fused=True, call="graph"),
        # Three MoE layers of a 256-token canvas, 128 experts top-8: router logits in, input already quantised by the
        # kernel in front, GeGLU.
        dict(name="moe_canvas", kind="moe", rows=256, hidden=2816, f=704, experts=128, top_k=8, layers=3, routing="uniform",
             activation="geglu", shared=False, router=True, fused=True, call="graph"),
        # A handful of tokens on a small expert set, called from Python without a group: odd row count, latency.
        dict(name="moe_few", kind="moe", rows=7, hidden=2048, f=512, experts=64, top_k=8, layers=1, routing="uniform",
             activation="swiglu", shared=False, router=False, fused=False, call="eager"),
        # A whole block in the device loop: begin, eight rounds of four layers (o_proj + norm, shared expert, routed
        # experts + norm) with the row statistics gathered at the end of each round, commit.
        dict(name="block_loop", kind="block", rows=32, hidden=2048, k_o=2048, f=512, experts=64, top_k=8, layers=4, rounds=8),
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "dense", "dense", "reduce", "moe", "moe", "moe", "block"])
    if kind == "linear":
        n = _log(rng, 128, 8192, 128)
        return dict(kind=kind, rows=_log(rng, 16, 256, 16), n=n, k=_log(rng, 64, min(151936, 388956160 // n), 8),
                    nn=rng.random() < 0.3)
    if kind == "dense":
        return dict(kind=kind, rows=_log(rng, 16, 256, 16), hidden=256 * rng.randint(2, 12), k_o=_log(rng, 256, 8192, 8),
                    k_d=_log(rng, 256, 9728, 8), layers=rng.randint(1, 8), call=rng.choice(["graph", "graph", "eager"]))
    if kind == "reduce":
        return dict(kind=kind, rows=rng.randint(1, 256), hidden=_log(rng, 256, 8192, 256), pairs=rng.randint(1, 8),
                    call=rng.choice(["graph", "eager"]))
    if kind == "block":
        return dict(kind=kind, rows=16 * rng.randint(1, 4), hidden=256 * rng.randint(4, 10), k_o=_log(rng, 512, 4096, 8),
                    f=64 * rng.randint(4, 8), experts=rng.choice([16, 32, 64]), top_k=rng.randint(2, 8),
                    layers=rng.randint(1, 4), rounds=rng.randint(1, 8))
    fused = rng.random() < 0.6  # a fused call site may not run twice in a row: a model has at least two
    experts = rng.choice([8, 16, 32, 64, 128, 256])
    return dict(kind=kind, rows=_log(rng, 1, 256, 1), hidden=256 * rng.randint(4, 11), f=64 * rng.randint(4, 11),
                experts=experts, top_k=rng.randint(1, 8), layers=rng.randint(2 if fused else 1, 3),
                routing=rng.choice(["uniform", "zipf"]), activation=rng.choice(["swiglu", "geglu"]),
                shared=rng.random() < 0.5, router=rng.random() < 0.3, fused=fused,
                call=rng.choice(["graph", "graph", "eager"]))


# -- inputs --------------------------------------------------------------------------------------------------------------
def _normal(g, *shape, std=1.0, mean=0.0):
    return torch.empty(*shape, device=DEVICE, dtype=torch.bfloat16).normal_(mean, std, generator=g)


def _popularity(case):
    """Relative popularity of the experts: even, or Zipf(1.2)."""
    e = torch.arange(1, case["experts"] + 1, dtype=torch.float64)
    p = e ** -1.2 if case.get("routing") == "zipf" else torch.ones_like(e)
    return p / p.sum()


def _router_logits(g, case):
    """Router logits ~ N(0, 1) per token, on top of the experts' popularity (Gumbel noise, so that the top-k is a draw
    without replacement from it)."""
    e = case["experts"]
    if case.get("routing") != "zipf":
        return _normal(g, case["rows"], e)
    p = _popularity(case).to(DEVICE)[torch.randperm(e, generator=g, device=DEVICE)]
    u = torch.rand(case["rows"], e, generator=g, device=DEVICE, dtype=torch.float64).clamp_min(1e-12)
    return (p.log() - (-u.log()).log()).to(torch.bfloat16)


def _packed(g, case):
    """A packed top-k as a model's own router hands it over: experts ascending, BF16 weights that sum to about 2.5."""
    top = _router_logits(g, case).float().topk(case["top_k"], dim=-1)
    ids, order = top.indices.sort(-1)
    weights = torch.softmax(top.values, -1).gather(1, order) * 2.5
    return nvfp4.pack(ids.int(), weights).contiguous()


def _experts(g, case, group):
    """One layer's NVFP4 experts from checkpoint tensors: weights of standard deviation near 0.02, input scales for
    activations of order one."""
    e, hidden, f = case["experts"], case["hidden"], case["f"]
    parts = {}
    scale2 = torch.tensor(0.0053, device=DEVICE)
    for proj, n, k, a in (("gate", f, hidden, 0.0019), ("up", f, hidden, 0.0019), ("down", hidden, f, 0.003)):
        codes = torch.randint(0, 256, (e, n, k // 2), generator=g, device=DEVICE, dtype=torch.uint8)
        scales = torch.randint(0x34, 0x3E, (e, n, k // 16), generator=g, device=DEVICE, dtype=torch.uint8)
        scales = scales.view(torch.float8_e4m3fn)
        a = torch.tensor(a, device=DEVICE)
        for i in range(e):
            parts[0, i, proj, "weight"], parts[0, i, proj, "weight_scale"] = codes[i], scales[i]
            parts[0, i, proj, "weight_scale_2"], parts[0, i, proj, "input_scale"] = scale2, a
    return nvfp4.b200_experts(parts, 0, 0, e, DEVICE, group=group)


def _capture(body, passes=2, keep=False):
    """`body` run eagerly `passes` times (buffers come into being), then captured once."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(passes):
            body()
        graph = torch.cuda.CUDAGraph(keep_graph=True) if keep else torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = body()
    torch.cuda.current_stream().wait_stream(stream)
    return graph, out


def _state(body, call):
    """What `run` needs: the Python calls themselves, or their captured graph and what the calls returned."""
    if call == "eager":
        return SimpleNamespace(body=body, graph=None)
    graph, out = _capture(body)
    return SimpleNamespace(body=body, graph=graph, out=out)


# -- the kinds -----------------------------------------------------------------------------------------------------------
def _prepare_linear(case, g):
    rows, n, k = case["rows"], case["n"], case["k"]
    if case["nn"]:  # y = probabilities @ embedding
        layer = Linear(_normal(g, k, n, std=0.02), nn=True)
        x = torch.softmax(_normal(g, rows, k, std=3.0), -1)
    else:
        layer = Linear(_normal(g, n, k, std=0.02))
        x = _normal(g, rows, k)
    out = torch.empty(rows, n, device=DEVICE, dtype=torch.bfloat16)
    return _state(lambda: layer(x, out=out), "eager")


def _prepare_dense(case, g):
    rows, hidden = case["rows"], case["hidden"]
    group = Group.local(DEVICE)
    x = [_normal(g, rows, k) for k in (case["k_o"], case["k_d"])]
    h = _normal(g, rows, hidden)
    layers = [([Linear(_normal(g, hidden, k, std=0.02), group=group) for k in (case["k_o"], case["k_d"])],
               [_normal(g, hidden, std=0.1, mean=1.0) for _ in range(2)]) for _ in range(case["layers"])]

    def body():
        for i, (linears, norms) in enumerate(layers):
            p = linears[0](x[0], out=group.partial(f"{i}.o", (rows, hidden)))
            group.reduce_norm(p, h, norms[0], EPS, site=f"{i}.post", replicated=rows <= 64)
            p = linears[1](x[1], out=group.partial(f"{i}.down", (rows, hidden)))
            out = group.reduce_norm(p, h, norms[1], EPS, site=f"{i + 1}.input", replicated=rows <= 64)
        return out, h

    return _state(body, case["call"])


def _prepare_reduce(case, g):
    rows, hidden = case["rows"], case["hidden"]
    group = Group.local(DEVICE)
    given = [_normal(g, rows, hidden) for _ in range(2 * case["pairs"])]
    norms = [_normal(g, hidden, std=0.1, mean=1.0) for _ in range(case["pairs"])]
    h = _normal(g, rows, hidden)

    def body():
        for i in range(case["pairs"]):
            group.reduce_norm(given[2 * i], h, norms[i], EPS, site=f"{i}.norm")
            out = group.reduce(given[2 * i + 1], site=f"{i}.sum")
        return out, h

    return _state(body, case["call"])


def _prepare_moe(case, g):
    rows, hidden, f, e = case["rows"], case["hidden"], case["f"], case["experts"]
    group = Group.local(DEVICE) if case["fused"] else None
    layers = [_experts(g, case, group) for _ in range(case["layers"])]
    x = _normal(g, rows, hidden)
    shared = _normal(g, rows, hidden) if case["shared"] else None
    outs = [torch.empty(rows, hidden, device=DEVICE, dtype=torch.bfloat16) for _ in layers]
    if case["router"]:
        config = SimpleNamespace(top_k_experts=case["top_k"], hidden_size=hidden, num_experts=e, moe_intermediate_size=f)
        experts = nvfp4.Experts(config, 0, rows, DEVICE)
        # The kernel in front leaves the layer's input quantised: codes and E4M3 block scales of activations of order one.
        experts.codes.copy_(torch.randint(0, 256, experts.codes.shape, generator=g, device=DEVICE, dtype=torch.uint8))
        experts.scales.copy_(torch.randint(0x68, 0x70, experts.scales.shape, generator=g, device=DEVICE, dtype=torch.uint8))
        logits = [_router_logits(g, case) for _ in layers]
        routed = [dict(fp4=layer, expert_scale=_normal(g, e, std=0.05, mean=1.0)) for layer in layers]
    else:
        packed = [_packed(g, case) for _ in layers]

    norms = [_normal(g, hidden, std=0.1, mean=1.0) for _ in layers]
    h = _normal(g, rows, hidden)

    def body():
        for i, layer in enumerate(layers):
            out = group.partial(f"{i}.moe", (rows, hidden)) if group is not None else outs[i]
            if case["router"]:
                out = experts(None, logits[i], routed[i], out)
            else:
                out = nvfp4.trtllm_moe(x, packed[i], layer, out, e, 0, f, activation=case["activation"], shared=shared)
            if group is not None and case["router"]:
                out = group.reduce(out, site=f"{i}.moe")
            elif group is not None:
                out = group.reduce_norm(out, h, norms[i], EPS, site=f"{i + 1}.input", replicated=True)
        if group is None:
            return outs, experts.packed if case["router"] else None
        return out, experts.packed if case["router"] else h

    return _state(body, case["call"])


def _prepare_block(case, g):
    rows, hidden, f, e = case["rows"], case["hidden"], case["f"], case["experts"]
    group = Group.local(DEVICE)
    layers = [SimpleNamespace(o=Linear(_normal(g, hidden, case["k_o"], std=0.02), group=group),
                              shared=Linear(_normal(g, hidden, f, std=0.02)), experts=_experts(g, case, group),
                              packed=_packed(g, case),
                              norms=[_normal(g, hidden, std=0.1, mean=1.0) for _ in range(2)])
              for _ in range(case["layers"])]
    attention, hidden_act = _normal(g, rows, case["k_o"]), _normal(g, rows, f)
    h0 = _normal(g, rows, hidden)
    h, shared = torch.empty_like(h0), torch.empty_like(h0)
    final = torch.empty(1, rows, 4, device=DEVICE)
    stats = torch.empty(rows, 4, device=DEVICE)
    x = torch.empty_like(h0)
    remaining, step = (torch.zeros(1, device=DEVICE, dtype=torch.int32) for _ in range(2))

    def begin():
        h.copy_(h0)
        remaining.fill_(case["rounds"])
        step.zero_()

    def round_():
        for i, layer in enumerate(layers):
            p = layer.o(attention, out=group.partial(f"{i}.o", (rows, hidden)))
            normed = group.reduce_norm(p, h, layer.norms[0], EPS, site=f"{i}.post", replicated=True)
            layer.shared(hidden_act, out=shared)
            p = nvfp4.trtllm_moe(normed, layer.packed, layer.experts, group.partial(f"{i}.moe", (rows, hidden)), e, 0, f,
                                 activation="swiglu", shared=shared)
            out = group.reduce_norm(p, h, layer.norms[1], EPS, site=f"{i + 1}.input", replicated=True)
        x.copy_(out)
        stats.copy_(x[:, :4])
        gathered = group.all_gather(stats, "stats")
        remaining.sub_(1)
        step.add_(1)
        return gathered

    def commit():
        final.copy_(group.symmetric("stats", (1, rows, 4), torch.float32))

    graphs = [_capture(fn, keep=True)[0] for fn in (begin, round_, commit)]
    block = BlockGraph(*(graph.raw_cuda_graph() for graph in graphs), remaining.data_ptr(), step.data_ptr(), case["rounds"])
    return SimpleNamespace(block=block, graphs=graphs, keep=(layers, attention, hidden_act, h0, shared, stats, group),
                           words=(remaining, step), out=(x, h, final, remaining, step))


_PREPARE = {"linear": _prepare_linear, "dense": _prepare_dense, "reduce": _prepare_reduce, "moe": _prepare_moe,
            "block": _prepare_block}


def prepare(case, seed):
    torch.cuda.set_device(DEVICE)
    return _PREPARE[case["kind"]](case, torch.Generator(device=DEVICE).manual_seed(seed))


def run(state):
    if hasattr(state, "block"):
        state.block.replay(torch.cuda.current_stream().cuda_stream)
        return state.out
    if state.graph is None:
        return state.body()
    state.graph.replay()
    return state.out


# -- what a pass cannot do without ---------------------------------------------------------------------------------------
def _active_experts(case):
    """Expected number of experts that a block's tokens reach. Drawing k of E without replacement by popularity p takes
    expert i with probability 1 - exp(-t p_i), t such that these sum to k."""
    p = _popularity(case)
    lo, hi = 0.0, 1e9
    for _ in range(200):
        t = (lo + hi) / 2
        if float((1 - torch.exp(-t * p)).sum()) < min(case["top_k"], case["experts"] - 1e-6):
            lo = t
        else:
            hi = t
    return float((1 - torch.exp(-lo * p) ** case["rows"]).sum())


def _moe_layer(case):
    """(bytes, flops) of one routed-expert layer: the active experts' codes and scales once, the input and the output."""
    rows, hidden, f = case["rows"], case["hidden"], case["f"]
    weights = _active_experts(case) * 3 * hidden * f * 9 / 16
    rows_in = rows * hidden * (9 / 16 if case.get("router") else 2)
    routing = rows * (case["experts"] * 2 if case.get("router") else case["top_k"] * 4)
    return weights + rows_in + routing + rows * hidden * 2, 2.0 * rows * case["top_k"] * 3 * hidden * f


def work(case):
    kind, rows = case["kind"], case["rows"]
    if kind == "linear":
        n, k = case["n"], case["k"]
        return {"bytes": 2.0 * (n * k + rows * k + rows * n), "flops": 2.0 * rows * n * k}
    hidden = case["hidden"]
    block = 2.0 * rows * hidden
    if kind == "reduce":  # partials read, residual stream read and written once, the last result and the norms
        return {"bytes": case["pairs"] * 2 * block + 3 * block + case["pairs"] * 2 * hidden,
                "flops": case["pairs"] * 6.0 * rows * hidden}
    if kind == "dense":
        k = case["k_o"] + case["k_d"]
        return {"bytes": case["layers"] * 2.0 * hidden * (k + 2) + 2.0 * rows * k + 3 * block,
                "flops": case["layers"] * 2.0 * rows * hidden * k}
    if kind == "moe":
        nbytes, flops = _moe_layer(case)
        shared = block if case["shared"] else 0
        return {"bytes": case["layers"] * nbytes + shared, "flops": case["layers"] * flops}
    nbytes, flops = _moe_layer(case)
    dense = hidden * (case["k_o"] + case["f"])
    passes = case["rounds"] * case["layers"]
    return {"bytes": passes * (nbytes + 2.0 * dense) + 3 * block, "flops": passes * (flops + 2.0 * rows * dense)}


def tolerance(case):
    """BF16 results of FP32 sums: 1e-2. The routed experts round their hidden activations to four bits in between, where
    another order of summation moves a value by a whole step now and then: 2e-2."""
    if case["kind"] in ("moe", "block"):
        return {"rel": 2e-2, "max": 0.5, "differ": 5e-3}
    return {"rel": 1e-2, "max": 0.1}
