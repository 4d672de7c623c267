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


# first and last slot of a token, of a block, negative and too large; the range of int32 exceeded
@pytest.mark.parametrize("at,expert", [((0, 0), -1), ((1023, 1), 8), ((511, 1), 2 ** 33), ((1299, 0), -2 ** 40)])
def test_an_expert_outside_the_range_is_reported_and_reads_nothing(at, expert):
    from sharq_b200 import ops

    tokens, experts, width = 1300, 8, 64
    selected = torch.rand(tokens, experts, generator=torch.Generator().manual_seed(1)).topk(2, dim=1).indices.cuda()
    good_dest = ops.moe_plan(selected, experts)[0]
    selected[at] = expert
    dest, src_row, _ = ops.moe_plan(selected, experts)
    with pytest.raises(RuntimeError, match="expert id"):
        ops.check_device_errors()
    ops.check_device_errors()  # reported once
    assert int(dest[at]) == -1 and int((dest < 0).sum()) == 1 and int(good_dest.min()) >= 0
    valid = dest >= 0
    assert torch.equal(src_row[dest[valid].long()].long(), valid.nonzero()[:, 0])
    y = torch.ones(src_row.numel(), width, dtype=torch.bfloat16, device="cuda")
    out = ops.moe_combine(y, dest, selected, torch.full((tokens, 2), 0.5, dtype=torch.bfloat16, device="cuda"))
    bad = torch.zeros(tokens, dtype=torch.bool, device="cuda")
    bad[at[0]] = True
    assert torch.equal(out.isnan().all(dim=1), bad) and bool((out[~bad] == 1).all())
