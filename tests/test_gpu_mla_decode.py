"""Decode attention of the latent cache on tcgen05 (csrc/mla_decode.cu) against fp32: head counts, tile edges, shares of the keys, a
moving maximum."""
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import mla

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("lens", [[1], [63], [64, 65], [1, 128, 129, 1000, 2, 64], [3000, 5]])
@pytest.mark.parametrize("h", [8, 16, 40, 128, 130])
@pytest.mark.parametrize("splits,grow", [(0, False), (1, True), (5, True)])
def test_matches_fp32(lens, h, splits, grow, monkeypatch):
    B, nope = len(lens), 128
    if splits:
        monkeypatch.setattr(mla, "mla_decode_splits", lambda *a: splits)
    g = torch.Generator(device="cuda").manual_seed(h)
    n = sum(lens)
    kv = torch.randn(n + 2, 1, 576, device="cuda", generator=g)
    q_lat = torch.randn(B, h, 512, device="cuda", generator=g).to(BF)
    q3 = torch.randn(B, h, nope + 64, device="cuda", generator=g).to(BF)
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(1)).to(torch.int32)
    r2t = torch.zeros(B + 2, max(lens) + 3, dtype=torch.int32)
    at = 0
    for b, L in enumerate(lens):
        r2t[b + 1, :L] = perm[at:at + L]
        if grow:     # scores that grow along the context
            kv[perm[at:at + L].long().cuda()] *= torch.linspace(0.05, 1.5, L, device="cuda").view(-1, 1, 1)
        at += L
    kv[n:] = float("nan")
    kv = kv.to(BF)
    rows = torch.arange(1, B + 1, dtype=torch.int32, device="cuda")
    seq = torch.tensor(lens, dtype=torch.int32, device="cuda")
    cu = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    scale = 0.1 if grow else 192 ** -0.5
    got = mla.mla_attention(q_lat, q3[:, :, nope:], kv, r2t.cuda(), rows, seq, cu, seq - 1, 512, scale, False, 1, max(lens)).float()
    want = mla.ref_mla_attention(q_lat.float(), q3[:, :, nope:].float(), kv, r2t.cuda(), rows.cpu(), seq.cpu(), cu.cpu(), (seq - 1).cpu(),
                                 512, scale)
    # weights rounded to bf16 and one rounding of values of up to about 5
    err = (got - want).abs().max().item()
    assert err < 4e-2, (err, [(got - want)[i].abs().max().item() for i in range(B)])
    assert int(ops.gemm_status("cuda:0").item()) == 0


@pytest.mark.parametrize("B", [1, 96])
@pytest.mark.parametrize("first", [0, 32, 64, 96])
def test_one_warp_rescales(B, first):
    """The maximum of 32 heads (a warp's rows) moves in every tile, that of the others never: a warp that is a tile ahead must not be
    counted for the one that lags."""
    L, h, nope, a = 3000, 128, 128, 6.8    # scores grow by 590 (as powers of two) over 47 tiles: 12.6 a tile, the threshold is 8
    g = torch.Generator(device="cuda").manual_seed(first)
    sign = torch.randint(0, 2, (576,), device="cuda", generator=g).float() * 2 - 1
    kv = torch.linspace(0.05, 1.5, L, device="cuda")[:, None] * sign + 0.1 * torch.randn(L, 576, device="cuda", generator=g)
    kv = kv.view(L, 1, 576).to(BF)
    q = 0.05 * torch.randn(B, h, 576, device="cuda", generator=g)
    q[:, first:first + 32] = a * sign
    q_lat = q[:, :, :512].to(BF).contiguous()
    q3 = torch.zeros(B, h, nope + 64, device="cuda", dtype=BF)
    q3[:, :, nope:] = q[:, :, 512:].to(BF)
    r2t = torch.arange(L, dtype=torch.int32, device="cuda").expand(B, L).contiguous()
    rows = torch.arange(B, dtype=torch.int32, device="cuda")
    seq = torch.full((B,), L, dtype=torch.int32, device="cuda")
    cu = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    f = lambda: mla.mla_attention(q_lat, q3[:, :, nope:], kv, r2t, rows, seq, cu, seq - 1, 512, 192 ** -0.5, False, 1, L)  # noqa: E731
    outs = [f() for _ in range(4)]
    s = torch.einsum("bhd,ld->bhl", torch.cat([q_lat, q3[:, :, nope:]], 2).double(), kv[:, 0].double()) * 192 ** -0.5
    want = torch.einsum("bhl,ld->bhd", torch.softmax(s, -1), kv[:, 0, :512].double())
    assert (outs[0].double() - want).abs().max().item() < 2e-2   # weights and outputs (up to 1.8) rounded to bf16
    assert all(torch.equal(outs[0], o) for o in outs)
    assert int(ops.gemm_status("cuda:0").item()) == 0


@pytest.mark.parametrize("keys,spread", [(300, 2.5), (300, 4.0), (1000, 2.5), (200, 1.0)])
def test_error_of_sharp_scores(keys, spread, monkeypatch):
    """As for prompt attention: the error against 64 bits is that of a pass in 64 bits with an exact running maximum."""
    from test_gpu_prompt_attention import running_softmax

    monkeypatch.setattr(mla, "mla_decode_splits", lambda *a: 1)
    B, h = 8, 128
    g = torch.Generator(device="cuda").manual_seed(keys)
    kv = torch.randn(B * keys, 1, 576, device="cuda", generator=g).to(BF)
    q = (torch.randn(B, h, 576, device="cuda", generator=g) * spread).to(BF)
    q_lat, q3 = q[:, :, :512].contiguous(), torch.nn.functional.pad(q[:, :, 512:], (128, 0))
    r2t = torch.arange(B * keys, dtype=torch.int32, device="cuda").view(B, keys)
    i = torch.arange(B + 1, dtype=torch.int32, device="cuda")
    seq = torch.full((B,), keys, dtype=torch.int32, device="cuda")
    got = mla.mla_attention(q_lat, q3[:, :, 128:], kv, r2t, i[:B], seq, i, seq - 1, 512, 576 ** -0.5, False, 1, keys)
    rows = kv.view(B, keys, 576).double()
    s = q.double() @ rows.transpose(1, 2) * 576 ** -0.5
    want = torch.softmax(s, -1) @ rows[:, :, :512]
    err = lambda x: ((x - want).norm() / want.norm()).item()  # noqa: E731
    assert err(got.double()) <= 1.05 * err(running_softmax(s, rows[:, :, :512], 64).float().to(BF).double())
