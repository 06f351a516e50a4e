"""Host side of the routed experts without a GPU: what `trtllm_moe` hands to the library, through a stand-in for it."""

from types import SimpleNamespace

import pytest
import torch

from dlmrt_b200 import _lib
from dlmrt_b200.quantization import nvfp4

ROWS, HIDDEN, F, EXPERTS = 8, 256, 128, 8


class FakeLibrary:
    """Keeps the descriptors of the launches; the sizes come from the real library."""

    def __init__(self):
        self.front, self.back = [], []
        self.dlm_moe_workspace_bytes = _lib.lib().dlm_moe_workspace_bytes

    def dlm_moe_front_nvfp4(self, f, pdl, stream):
        self.front.append(type(f).from_buffer_copy(f))
        return _lib.OK

    def dlm_moe_nvfp4(self, m, out, ldo, pdl, stream):
        self.back.append(type(m).from_buffer_copy(m))
        return _lib.OK


@pytest.fixture
def library(monkeypatch):
    fake = FakeLibrary()
    monkeypatch.setattr(nvfp4, "_lib", SimpleNamespace(lib=lambda: fake, stream=lambda t: 0, check=_lib.check))
    return fake


def make_experts(count=EXPERTS):
    parts = {}
    for e in range(count):
        for proj, n, k in (("gate", F, HIDDEN), ("up", F, HIDDEN), ("down", HIDDEN, F)):
            parts[0, e, proj, "weight"] = torch.zeros(n, k // 2, dtype=torch.uint8)
            parts[0, e, proj, "weight_scale"] = torch.zeros(n, k // 16, dtype=torch.uint8)
            parts[0, e, proj, "weight_scale_2"] = parts[0, e, proj, "input_scale"] = torch.tensor(1.0)
    return nvfp4.b200_experts(parts, 0, 0, count, "cpu")


def call(experts, top_k, num_experts=EXPERTS, packed_rows=ROWS):
    x = torch.zeros(ROWS, HIDDEN, dtype=torch.bfloat16)
    packed = torch.zeros(packed_rows, top_k, dtype=torch.int32)
    nvfp4.trtllm_moe(x, packed, experts, torch.empty_like(x), num_experts, 0, F)


def test_calls_of_other_top_k_or_expert_count_have_buffers_of_their_own(library):
    """The list length and the expert count size the scratch as the row count does: both halves of a call have to agree on
    them, and everything the device writes has to lie in memory sized for them, in whatever order the calls come. What
    a call used once stays where it is, since a captured graph may hold it."""
    experts = make_experts()
    for top_k, num_experts in ((2, 8), (6, 8), (2, 40), (2, 8), (6, 40)):
        call(experts, top_k, num_experts)
        f, m = library.front[-1], library.back[-1]
        assert (f.m, f.top_k, f.e_total) == (ROWS, top_k, num_experts) == (m.m, m.top_k, m.e_total)
        assert (f.ids, f.weights, f.counts, f.amap) == (m.ids, m.weights, m.counts, m.amap)
        elements = {t.data_ptr(): t.numel() for b in experts["_buffers"].values() for t in (b.ids, b.weights, b.counts, b.amap)}
        assert elements[f.ids] == elements[f.weights] == ROWS * top_k
        assert elements[f.counts] == num_experts and elements[f.amap] == num_experts * f.m_max
        assert m.workspace_bytes >= library.dlm_moe_workspace_bytes(ROWS, HIDDEN, top_k)
    assert library.front[0].ids == library.front[3].ids  # the first call's buffers again


def test_a_top_k_list_of_too_few_rows_is_refused(library):
    with pytest.raises(ValueError, match="packed"):
        call(make_experts(), 2, packed_rows=ROWS - 1)
    assert not library.front
