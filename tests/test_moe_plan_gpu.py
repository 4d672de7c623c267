"""The grouping plan of a mixture-of-experts step in two launches against the ATen composition on the CPU."""
import pytest
import torch

from sharq_b200.decoder import moe_grouping

pytestmark = pytest.mark.gpu


# one token, one block and one more slot, several blocks with a ragged last, one expert, all slots on one expert
@pytest.mark.parametrize("tokens,experts,top_k", [(1, 8, 2), (512, 8, 2), (513, 8, 2), (5000, 16, 3), (700, 1, 1), (1300, 4, 1)])
def test_plan_equals_the_aten_plan(tokens, experts, top_k):
    g = torch.Generator().manual_seed(tokens)
    selected = torch.rand(tokens, experts, generator=g).topk(top_k, dim=1).indices
    if experts == 4:
        selected[:] = 2
    want = moe_grouping(selected, experts)
    got = moe_grouping(selected.cuda(), experts)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a.cpu(), b)
