"""Prompt attention with scores and outputs in tensor memory (csrc/attention_fa.cu) against fp32: edges of the query and key tiles,
cached prefixes, ragged batches, odd head groups, moving maxima, strided queries."""
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import reference as ref
from lightllm_b200.ops._native import kernels

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
CASES = [([1], [0]), ([127], [1]), ([128], [128]), ([129, 1, 300], [0, 700, 127]), ([256, 257], [0, 3]), ([37, 5, 640], [600, 0, 129]),
         ([383], [2000])]


def _run(new, ready, Hq, Hkv, scale=1.0, seed=0, grow=None, pad=0):
    D, B, T = 128, len(new), sum(new)
    g = torch.Generator(device="cuda").manual_seed(seed)
    lens = [a + b for a, b in zip(new, ready)]
    n = sum(lens)
    kv = torch.randn(n + 3, 2 * Hkv, D, device="cuda", generator=g)
    if grow is not None:   # scores that grow along the context: the running maximum has to move
        kv[:, :Hkv] *= grow
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(seed)).to(torch.int32)
    r2t = torch.zeros(B + 2, max(lens) + 1, dtype=torch.int32)
    at = 0
    for b, L in enumerate(lens):
        r2t[b + 1, :L] = perm[at:at + L]
        if grow is not None:
            kv[perm[at:at + L].long().cuda(), :Hkv] *= torch.linspace(0.05, 1.0, L, device="cuda").view(-1, 1, 1)
        at += L
    kv[n:] = float("nan")      # slots of no request
    kv = kv.to(BF)
    qfull = (torch.randn(T, (Hq + 2 * Hkv) * D + pad, device="cuda", generator=g) * scale).to(BF)
    q = qfull[:, : Hq * D]
    cu = torch.tensor([0] + torch.tensor(new).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    rows = torch.arange(1, B + 1, dtype=torch.int32, device="cuda")
    rd = torch.tensor(ready, dtype=torch.int32, device="cuda")
    got = ops.gqa_prefill(q, kv, r2t.cuda(), rows, cu, rd, Hq, Hkv, D, max(new)).float()
    want = ref.gqa_prefill(q.reshape(T, Hq, D).float(), kv.float(), r2t.cuda(), rows, cu, rd, Hq, Hkv, D).view(T, Hq, D).float()
    assert kernels().llb_attn_fa_status() == 0
    return got, want


@pytest.mark.parametrize("new,ready", CASES)
@pytest.mark.parametrize("Hq,Hkv", [(8, 2), (4, 4), (6, 2), (2, 1)])
def test_matches_fp32(new, ready, Hq, Hkv):
    got, want = _run(new, ready, Hq, Hkv, pad=64)
    # weights rounded to bf16 (2^-9 each, averaged over the row) and one rounding of values up to about 4
    assert (got - want).abs().max().item() < 2e-2


def test_one_tile_kernel(monkeypatch):
    """The kernel that LLB_ATTN_FA=0 selects."""
    monkeypatch.setattr(ops, "_ATTN_FA", False)
    got, want = _run([129, 1, 300], [0, 700, 127], 6, 2, pad=64)
    assert kernels().llb_attn_tc_status() == 0
    assert (got - want).abs().max().item() < 2e-2   # as above


@pytest.mark.parametrize("grow", [1.0, 30.0])
def test_moving_maximum(grow):
    got, want = _run([300, 128], [500, 0], 8, 2, scale=2.0, grow=grow)
    assert (got - want).abs().max().item() < 4e-2      # sharp softmax: single values of up to 4.5, two roundings of 2^-9


def running_softmax(s, v, tile):
    """s [.., n, keys], v [.., keys, d] in 64 bits: the sums of a tiled pass whose weights, relative to the largest score so far, are rounded
    to bf16, divided by the sum of the weights before rounding."""
    m = torch.full(s.shape[:-1] + (1,), float("-inf"), dtype=s.dtype, device=s.device)
    l, o = 0.0, 0.0
    for k in range(0, s.shape[-1], tile):
        top = torch.maximum(m, s[..., k:k + tile].amax(-1, keepdim=True))
        w, alpha = torch.exp(s[..., k:k + tile] - top), torch.exp(m - top)
        o, l, m = o * alpha + w.float().to(BF).double() @ v[..., k:k + tile, :], l * alpha + w.sum(-1, keepdim=True), top
    return o / l


@pytest.mark.parametrize("keys,spread", [(1000, 2.5), (1000, 4.0), (6000, 2.5), (300, 1.0)])
def test_error_of_sharp_scores(keys, spread):
    """The weight of a row's largest key is exact.  The error against 64 bits is that of the pass in 64 bits whose weights are rounded that
    way (and whose output is rounded once), up to what fp32 sums and the order of the rounding can add; a maximum that lags is a fifth
    to a quarter above."""
    new, H, D = 200, 4, 128
    g = torch.Generator(device="cuda").manual_seed(keys)
    kv = torch.randn(keys, 2 * H, D, device="cuda", generator=g).to(BF)
    q = (torch.randn(new, H * D, device="cuda", generator=g) * spread).to(BF)
    i = lambda *x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    got = ops.gqa_prefill(q, kv, torch.arange(keys, dtype=torch.int32, device="cuda").view(1, -1), i(0), i(0, new), i(keys - new), H, H, D, new)
    k, v = kv[:, :H].double().transpose(0, 1), kv[:, H:].double().transpose(0, 1)
    s = q.view(new, H, D).double().transpose(0, 1) @ k.transpose(1, 2) / D ** 0.5
    s.masked_fill_(torch.arange(keys, device="cuda")[None] > torch.arange(new, device="cuda")[:, None] + keys - new, float("-inf"))
    want = torch.softmax(s, -1) @ v
    err = lambda x: ((x - want).norm() / want.norm()).item()  # noqa: E731
    assert err(got.view(new, H, D).transpose(0, 1).double()) <= 1.05 * err(running_softmax(s, v, 128).float().to(BF).double())
