"""Split-K scratch that a captured graph may still be writing to outlives the call that needs a larger one."""

import weakref

import pytest
import torch

from gpu_util import assert_same_bits, bits, randn_bf16


def linear_scratch(monkeypatch):
    """Scratch of a Linear's own GEMM for `rows` rows, on the CPU: the launch itself goes to a stand-in."""
    from types import SimpleNamespace

    from dlmrt_b200 import _lib
    from dlmrt_b200.layers import linear

    seen = []
    fake = SimpleNamespace(dlm_workspace_bytes=_lib.lib().dlm_workspace_bytes,
                           dlm_gemm_bf16=lambda g, *rest: seen.append((g.workspace, g.workspace_bytes)) or 0)
    monkeypatch.setattr(linear, "_lib", SimpleNamespace(**{**vars(_lib), "lib": lambda: fake, "stream": lambda t: 0}))
    lin = linear.Linear(torch.zeros(2560, 512, dtype=torch.bfloat16))

    def call(rows):
        lin(torch.zeros(rows, 512, dtype=torch.bfloat16))
        return seen[-1]

    return lin, call


def tensors_of(owner):
    """Every tensor that `owner` holds, as weak references by address."""
    found, todo = {}, [vars(owner)]
    while todo:
        item = todo.pop()
        if isinstance(item, torch.Tensor):
            found[item.data_ptr()] = weakref.ref(item)
        elif isinstance(item, dict):
            todo += list(item.values())
        elif isinstance(item, (list, tuple)):
            todo += list(item)
    return found


def test_a_linear_keeps_the_scratch_it_has_outgrown(monkeypatch):
    lin, call = linear_scratch(monkeypatch)
    used = [call(rows) for rows in (16, 32, 256, 16)]
    held = tensors_of(lin)
    for address, nbytes in used:
        assert held[address]().numel() == nbytes, "scratch of an earlier call was given back"


def test_a_group_keeps_the_scratch_it_has_outgrown():
    from dlmrt_b200.distributed.parallel import Group

    g = Group.local("cpu")
    used = [(ws.data_ptr(), ws.numel()) for ws in (g.workspace(0, n) for n in (4096, 1 << 16, 1 << 20, 4096))]
    other = g.workspace(1, 4096)
    assert other.data_ptr() not in dict(used)  # another chain's calls may overlap in time
    held = tensors_of(g)
    for address, nbytes in used:
        assert held[address]().numel() == nbytes, "scratch of an earlier call was given back"
    assert sum(t().numel() for a, t in held.items() if a in dict(used)) <= 2 * used[-1][1]


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [False, True])
def test_a_captured_graph_survives_a_larger_eager_call(fused):
    """A graph captured at 32 rows, an eager call at 256 rows (which needs larger scratch), memory allocated and filled
    after it: the replay still gives the captured call's bits."""
    from dlmrt_b200.distributed.parallel import Group
    from dlmrt_b200.layers.linear import Linear

    n, k = 2048, 4096
    g = Group.local("cuda:0")
    lin = Linear(randn_bf16(n, k, seed=1, std=0.02), group=g)
    xs = {rows: randn_bf16(rows, k, seed=rows) for rows in (32, 256)}
    partials = {rows: g.symmetric(f"p{rows}", (rows, n)) for rows in xs}
    outs = {rows: torch.empty(rows, n, device="cuda", dtype=torch.bfloat16) for rows in xs}

    def call(rows):
        if not fused:
            return lin.gemm(xs[rows], outs[rows])
        g.reduce(lin(xs[rows], out=partials[rows]), site=f"a{rows}")
        return g.reduce(lin(xs[rows], out=partials[rows]), site=f"b{rows}")

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        want = bits(call(32))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            captured = call(32)
    torch.cuda.synchronize()
    call(256)
    torch.cuda.synchronize()
    junk = [torch.full((1 << 20,), 0x7F, device="cuda", dtype=torch.uint8) for _ in range(64)]
    captured.fill_(0)
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert_same_bits(bits(captured), want, "replay after a larger call")
    g.check()
    assert all(bool((t == 0x7F).all()) for t in junk), "the replay wrote into memory of other tensors"
