"""Prompt attention of the latent cache in its expanded form against fp32, and the rule that chooses between the forms."""
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import mla


def _ref(q, kv, pe, H, own, dv, cu_q, lens, ready, scale):
    T = q.shape[0]
    out = torch.zeros(T, H, dv, device=q.device)
    r0 = 0
    for b in range(len(lens)):
        s0, s1 = cu_q[b], cu_q[b + 1]
        L = lens[b]
        k = torch.cat([kv[r0:r0 + L, : H * own].view(L, H, own), pe[r0:r0 + L, None].expand(-1, H, -1)], -1).float()
        v = kv[r0:r0 + L, H * own:].view(L, H, dv).float()
        s = torch.einsum("nhd,lhd->hnl", q[s0:s1].view(-1, H, k.shape[-1]).float(), k) * scale
        see = torch.arange(L, device=q.device)[None] <= torch.arange(s1 - s0, device=q.device)[:, None] + ready[b]
        s.masked_fill_(~see, float("-inf"))
        out[s0:s1] = torch.einsum("hnl,lhd->nhd", torch.softmax(s, -1), v)
        r0 += L
    return out.view(T, H * dv)


@pytest.mark.gpu
@pytest.mark.parametrize("new,ready", [([1], [0]), ([128, 1, 127], [0, 63, 65]), ([129, 64, 300, 5], [0, 500, 1, 1000])])
@pytest.mark.parametrize("dv", [64, 128])
def test_expanded_attention(new, ready, dv):
    H, own, rope, lat = 6, 128, 64, 512
    g = torch.Generator(device="cuda").manual_seed(1)
    lens = [a + b for a, b in zip(new, ready)]
    rows, T = sum(lens), sum(new)
    q = torch.randn(T, H * (own + rope), device="cuda", generator=g).bfloat16()
    kv = torch.randn(rows, H * (own + dv), device="cuda", generator=g).bfloat16()
    c = torch.randn(rows, lat + rope, device="cuda", generator=g).bfloat16()
    cu = [0]
    for n in new:
        cu.append(cu[-1] + n)
    kr = mla.KeyRange(torch.tensor(ready), torch.tensor(new), 0, "cuda")
    out = torch.full((T, H * dv), 7.0, device="cuda", dtype=torch.bfloat16)
    scale = (own + rope) ** -0.5
    mla.latent_prefill(q, kv, c, lat, own, H, own + rope, dv, torch.tensor(cu, dtype=torch.int32, device="cuda"),
                       torch.tensor(ready, dtype=torch.int32, device="cuda"), kr, max(new), scale, out)
    want = _ref(q, kv, c[:, lat:], H, own, dv, cu, lens, ready, scale)
    # weights up to 2^-9 off (bf16 products), values of about 1, one rounding of the result
    assert (out.float() - want).abs().max().item() < 2e-2
    assert int(ops.gemm_status("cuda:0").item()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("new,ready", [([1, 100], [0, 0]), ([63, 1], [0, 64]), ([64, 64], [1, 0]), ([130, 70], [255, 3])])
def test_a_request_does_not_see_its_neighbour(new, ready, bad):
    """Keys and values of the requests lie back to back; the first one's output is what it is alone, whatever the second one holds."""
    H, own, rope, lat, dv = 3, 128, 64, 512, 128
    g = torch.Generator(device="cuda").manual_seed(5)
    first, rows, T = new[0] + ready[0], sum(new) + sum(ready), sum(new)
    q = torch.randn(T, H * (own + rope), device="cuda", generator=g).bfloat16()
    kv = torch.randn(rows, H * (own + dv), device="cuda", generator=g).bfloat16()
    c = torch.randn(rows, lat + rope, device="cuda", generator=g).bfloat16()
    kv[first:], c[first:] = bad, bad

    def run(n):
        t, r = sum(new[:n]), sum(new[:n]) + sum(ready[:n])
        cu = torch.tensor([0] + torch.tensor(new[:n]).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        kr = mla.KeyRange(torch.tensor(ready[:n]), torch.tensor(new[:n]), 0, "cuda")
        out = torch.empty((t, H * dv), device="cuda", dtype=torch.bfloat16)
        mla.latent_prefill(q[:t], kv[:r], c[:r], lat, own, H, own + rope, dv, cu, torch.tensor(ready[:n], dtype=torch.int32, device="cuda"),
                           kr, max(new[:n]), 0.1, out)
        return out[: new[0]]

    alone = run(1)
    assert alone.isfinite().all() and torch.equal(run(2), alone)


def test_rule(monkeypatch):
    t = torch.tensor
    row = 128 * 256 * 2
    assert mla.expanded_groups(t([1, 2]), t([5000, 100]), row) is None                # a few tokens behind long contexts
    assert mla.expanded_groups(t([300, 1500]), t([0, 1000]), row) == [(0, 2)]
    monkeypatch.setattr(mla, "EXPANDED_BYTES", 1000 * row)
    assert mla.expanded_groups(t([600, 400, 1, 999]), t([0, 0, 0, 0]), row) == [(0, 2), (2, 4)]
    assert mla.expanded_groups(t([600, 1001]), t([0, 0]), row) is None                # one request alone does not fit
