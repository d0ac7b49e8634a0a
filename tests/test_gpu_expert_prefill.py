"""Experts of a prompt pass: the cluster form of the sorted layout and the gather."""
import pytest
import torch

from lightllm_b200.ops import moe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _ids(T, E, k, seed, skew=False):
    g = torch.Generator().manual_seed(seed)
    p = torch.rand(T, E, generator=g)
    if skew:
        p[:, : max(1, E // 8)] += 0.7
        p[:, E // 2] = -1     # one expert without tokens
    return p.topk(k, -1).indices.to(torch.int32).cuda()


@pytest.mark.parametrize("T,E,k", [(511, 16, 8), (512, 16, 8), (4097, 3, 1), (8192, 128, 8), (700, 160, 6)])
@pytest.mark.parametrize("e0,skew", [(0, False), (0, True), (1, False)])
def test_layout(T, E, k, e0, skew):
    ids = _ids(T, E, k, T, skew)
    E_local = E - e0
    lay = moe.moe_align(ids, E_local, e0)
    flat = ids.view(-1).cpu() - e0
    sp, pr = lay.sorted_pair.cpu(), lay.pair_row.cpu()
    off, mb, total = lay.expert_off.cpu(), lay.mblock_expert.cpu(), int(lay.total_rows)
    want = torch.zeros(E_local + 1, dtype=torch.long)
    for e in range(E_local):
        n = int((flat == e).sum())
        want[e + 1] = want[e] + -(-n // 128) * 128
        rows = pr[flat == e]
        assert sorted(rows.tolist()) == list(range(int(want[e]), int(want[e]) + n))
    assert torch.equal(off.long(), want) and total == int(want[-1])
    assert (pr[flat < 0] == -1).all()
    live = sp >= 0
    assert int(live.sum()) == int((flat >= 0).sum()) and torch.equal(pr[sp[live].long()].long(), live.nonzero().view(-1))
    for b in range(lay.m_pad // 128):
        e = int(mb[b])
        assert (e == -1) == (b * 128 >= total)
        assert e < 0 or want[e] <= b * 128 < want[e + 1]
    x = torch.randn(T, 1024 + 8, device="cuda").to(BF)
    a = moe.gather_rows(x, lay)
    valid = sp[:total] >= 0
    assert torch.equal(a[:total][valid.cuda()], x[(sp[:total][valid] // k).long().cuda()]) and not a[:total][~valid.cuda()].any()
