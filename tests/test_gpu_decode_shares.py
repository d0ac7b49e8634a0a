"""Decode attention with shares of equal length over a ragged batch, and the rotary kernel's stores into 8-bit pools."""
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import kv_quant, reference as ref

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _batch(lens, seed=0):
    g = torch.Generator().manual_seed(seed)
    n = sum(lens)
    perm = torch.randperm(n, generator=g).to(torch.int32)
    r2t = torch.zeros(len(lens) + 3, max(lens) + 5, dtype=torch.int32)
    at = 0
    for b, L in enumerate(lens):
        r2t[b + 2, :L] = perm[at:at + L]
        at += L
    rows = torch.arange(2, len(lens) + 2, dtype=torch.int32)
    return n, r2t.cuda(), rows.cuda(), torch.tensor(lens, dtype=torch.int32).cuda()


RAGGED = [[1], [130], [5000], [1, 15, 16, 17, 3000, 127, 128, 129], [700] * 3 + [9000], list(range(1, 400, 3)), [2000] * 8 + [1] * 300]


@pytest.mark.parametrize("lens", RAGGED)
@pytest.mark.parametrize("kind", ["bf16", "int8", "fp8"])
@pytest.mark.parametrize("heads", [(8, 2), (32, 1)])
def test_ragged_batches(lens, kind, heads):
    Hq, Hkv = heads
    D, B = 128, len(lens)
    n, r2t, rows, b_len = _batch(lens)
    g = torch.Generator(device="cuda").manual_seed(3)
    kv = torch.randn(n, 2 * Hkv, D, device="cuda", generator=g).to(BF)
    q = torch.randn(B, Hq * D, device="cuda", generator=g).to(BF)
    slots = torch.arange(n, dtype=torch.int32, device="cuda")
    layer = kv
    if kind == "int8":
        layer = kv_quant.Int8KVLayer(torch.zeros(n, 2 * Hkv, D + 16, dtype=torch.int8, device="cuda"), D)
    elif kind == "fp8":
        layer = kv_quant.Fp8KVLayer(torch.zeros(n, 2 * Hkv, D, dtype=torch.uint8, device="cuda"), D,
                                    torch.linspace(0.01, 0.02, 2 * Hkv, device="cuda"))
    if kind != "bf16":
        kv_quant.quant_store_(layer, kv, slots)
        kv = layer.dequant_all(BF)
    want = ref.gqa_decode(q.view(B, Hq, D).float(), kv.float(), r2t, rows, b_len, Hq, Hkv, D).view(B, Hq, D).float()
    cap = ops.gqa_decode_num_splits(B, Hq, Hkv, max(lens))
    for splits in {1, 2, 5, 64, cap}:
        got = ops.gqa_decode(q, layer, r2t, rows, b_len, Hq, Hkv, D, max(lens), num_splits=splits).float()
        # 16-bit weights and values: 2^-8 of values up to about 4
        assert (got - want).abs().max().item() < 3e-2, splits


@pytest.mark.parametrize("D,rot", [(64, 64), (128, 128), (128, 64), (256, 256)])
@pytest.mark.parametrize("kind", ["int8", "fp8"])
@pytest.mark.parametrize("T,norm", [(1, False), (37, True)])
def test_fused_store_is_the_separate_one(D, rot, kind, T, norm):
    Hq, Hkv = 6, 3
    g = torch.Generator(device="cuda").manual_seed(T)
    qkv = (torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda", generator=g) * 3).to(BF)
    qkv[0, Hq * D:(Hq + 1) * D] = 0
    pos = torch.randint(0, 500, (T,), device="cuda", generator=g, dtype=torch.int32)
    slot = torch.randperm(T + 5, device="cuda", generator=g)[:T].to(torch.int32)
    cos, sin = torch.rand(512, rot // 2, device="cuda"), torch.rand(512, rot // 2, device="cuda")
    nw = [torch.rand(D, device="cuda").to(BF) for _ in range(2)] if norm else [None, None]

    def pool():
        if kind == "int8":
            return kv_quant.Int8KVLayer(torch.zeros(T + 5, 2 * Hkv, D + 16, dtype=torch.int8, device="cuda"), D)
        return kv_quant.Fp8KVLayer(torch.zeros(T + 5, 2 * Hkv, D, dtype=torch.uint8, device="cuda"), D,
                                   torch.linspace(0.004, 2.0, 2 * Hkv, device="cuda"))

    a, b = pool(), pool()
    q1, q2 = qkv.clone(), qkv.clone()
    ops.rope_kv_scatter_(q1, a, cos, sin, pos, slot, Hq, Hkv, D, rot, *nw)
    tmp = torch.empty(T, 2 * Hkv, D, dtype=BF, device="cuda")
    ops.rope_kv_scatter_(q2, tmp, cos, sin, pos, torch.arange(T, dtype=torch.int32, device="cuda"), Hq, Hkv, D, rot, *nw)
    kv_quant.quant_store_(b, tmp, slot)
    assert torch.equal(q1, q2) and torch.equal(a.data, b.data)


@pytest.mark.parametrize("lens", [[130] * 5, [256, 1, 17], list(range(16, 130, 4)), [2048, 3, 2047], [250] * 140 + [257] * 8, [255] * 147])
@pytest.mark.parametrize("fp8", [False, True])
def test_short_contexts(lens, fp8):
    """Batches whose requests get CTAs of their own, and their neighbours that are shared out."""
    Hq, Hkv, D, B = 8, 2, 128, len(lens)
    n, r2t, rows, b_len = _batch(lens)
    g = torch.Generator(device="cuda").manual_seed(4)
    kv = torch.randn(n, 2 * Hkv, D, device="cuda", generator=g).to(BF)
    q = torch.randn(B, Hq * D, device="cuda", generator=g).to(BF)
    layer = kv
    if fp8:
        layer = kv_quant.Fp8KVLayer(torch.zeros(n, 2 * Hkv, D, dtype=torch.uint8, device="cuda"), D, torch.full((2 * Hkv,), 0.01, device="cuda"))
        kv_quant.quant_store_(layer, kv, torch.arange(n, dtype=torch.int32, device="cuda"))
        kv = layer.dequant_all(BF)
    want = ref.gqa_decode(q.view(B, Hq, D).float(), kv.float(), r2t, rows, b_len, Hq, Hkv, D).view(B, Hq, D).float()
    for splits in (2, 3, 17, 64):
        got = ops.gqa_decode(q, layer, r2t, rows, b_len, Hq, Hkv, D, max(lens), num_splits=splits).float()
        assert (got - want).abs().max().item() < 3e-2, splits   # as above


def test_slots_of_partial_results():
    """Kernels that cut every context into equal parts get the number of parts that fills the GPU, others four times as many slots; a batch
    that fills the GPU by itself is not cut."""
    equal = lambda b, h, n: max(1, min(-(-592 // (b * h)), -(-n // 256), 64))  # noqa: E731
    for b, h, n in ((1, 8, 700), (4, 8, 4000), (64, 8, 2000), (74, 8, 2000), (100, 8, 1000), (592, 1, 5000), (600, 1, 300), (1183, 1, 9000)):
        parts = equal(b, h, n)
        assert ops.gqa_decode_num_splits(b, 4 * h, h, n, shares=False) == parts
        slots = ops.gqa_decode_num_splits(b, 4 * h, h, n)
        assert slots == 1 if parts == 1 else slots >= min(parts, 296 // h)
    assert not kv_quant.decode_shares(True, 64) and kv_quant.decode_shares(True, 128) and kv_quant.decode_shares(False, 64)
