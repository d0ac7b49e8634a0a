"""Few-token forms of the fp8 GEMM and of the experts (csrc/gemm_stream.cu) against fp32 on the same quantised operands."""
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import fp8, moe

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("M", [1, 16, 17, 48, 64, 65, 96, 128])
@pytest.mark.parametrize("N,K,epi,rows", [(1024, 1024, "store", 128), (1096, 1040, "store", 128), (4096, 7168, "residual", 128),
                                          (2304, 512, "gated_silu", 32), (256, 18432, "residual", 128)])
def test_fp8_dense(M, N, K, epi, rows):
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g).to(BF)
    w = fp8.Fp8Weight.from_float(torch.randn(N, K, device="cuda", generator=g) / K ** 0.5, rows)
    res = torch.randn(M, N, device="cuda", generator=g).to(BF) if epi == "residual" else None
    got = ops.gemm(x, w, epi=epi, residual=res).float()
    xq, xs = fp8.quant_act(x)
    want = fp8._epilogue_reference(fp8.dequant_act(xq, xs).double() @ w.dequant().double().t(), epi, res).float()
    # exact products of e4m3 values, fp32 sums, one rounding to bf16 (2^-9 of the value)
    assert ((got - want).abs() / want.abs().clamp_min(1.0)).max().item() < 2 ** -8
    assert int(ops.gemm_status("cuda:0").item()) == 0


def _route(T, E, k, seed, hot):
    g = torch.Generator().manual_seed(seed)
    if hot:   # everyone picks expert 1
        ids = torch.stack([torch.cat([torch.tensor([1]), torch.randperm(E - 2, generator=g)[: k - 1] + 2]) for _ in range(T)])
    else:
        ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    w = torch.rand(T, k, generator=g)
    return ids.to(torch.int32).cuda(), (w / w.sum(-1, keepdim=True)).cuda()


@pytest.mark.parametrize("T", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("kind", ["bf16", "bf16 gelu", "fp8"])
@pytest.mark.parametrize("hot,e0", [(False, 0), (True, 0), (False, 4)])
def test_experts(T, kind, hot, e0):
    E, k, H, I = 12, 4, 1024, 384
    E_local = E - e0
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H + 64, device="cuda", generator=g).to(BF)[:, :H]
    w13 = (torch.randn(E_local, 2 * I, H, device="cuda", generator=g) / H ** 0.5).to(BF)
    w2 = (torch.randn(E_local, H, I, device="cuda", generator=g) / I ** 0.5).to(BF)
    ids, wt = _route(T, E, k, T, hot)
    act = "gelu" if "gelu" in kind else "silu"
    r13, r2 = w13, w2
    if kind == "fp8":
        w13 = fp8.Fp8Experts(fp8.stack_experts([fp8.Fp8Weight.from_float(w.float(), 32) for w in w13]), E_local)
        w2 = fp8.Fp8Experts(fp8.stack_experts([fp8.Fp8Weight.from_float(w.float(), 128) for w in w2]), E_local)
        r13, r2 = w13.dequant().to(BF), w2.dequant().to(BF)
    out0 = torch.randn(T, H, device="cuda", generator=g).to(BF)
    got = moe.fused_experts(x, w13, w2, ids, wt, act, e0, out=out0.clone(), accumulate=True).float()
    want = out0.float() + moe.ref_fused_experts(x.cpu(), r13.cpu(), r2.cpu(), ids.cpu(), wt.cpu(), act, e0).cuda().float()
    # bf16: roundings of the gate and of every expert's output (2^-9 of values of about 1); fp8: activations quantised twice,
    # 2^-4 per element, averaged over the sums
    assert (got - want).abs().max().item() < (3e-2 if kind != "fp8" else 0.25)
    few, moe.FEW_TOKENS = moe.FEW_TOKENS, 0
    try:
        other = moe.fused_experts(x, w13, w2, ids, wt, act, e0, out=out0.clone(), accumulate=True).float()
    finally:
        moe.FEW_TOKENS = few
    # the other form: the same quantised operands, sums in another order
    assert (got - other).abs().max().item() < 3e-2
    assert int(ops.gemm_status("cuda:0").item()) == 0
