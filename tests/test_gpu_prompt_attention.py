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


@pytest.mark.parametrize("grow", [1.0, 30.0])
def test_moving_maximum(grow):
    got, want = _run([300, 128], [500, 0], 8, 2, scale=2.0, grow=grow)
    assert (got - want).abs().max().item() < 4e-2      # sharp softmax: single values of up to 4.5, two roundings of 2^-9
