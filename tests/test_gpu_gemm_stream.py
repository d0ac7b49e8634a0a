"""The few-token GEMM (csrc/gemm_stream.cu) against fp32: edges of the token tiles, ragged right edges, K tails, shares of K."""
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _case(M, N, K, epi, seed=0, pitch=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(M, K + pitch, device="cuda", generator=g).bfloat16()[:, :K]
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    res = torch.randn(M, N, device="cuda", generator=g).bfloat16() if epi == "residual" else None
    return a, w, res


@pytest.mark.parametrize("M", [1, 15, 16, 17, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("N,K,epi", [(1024, 1024, "store"), (1096, 1032, "store"), (4096, 4096, "residual"), (28672, 1024, "gated_silu"),
                                     (1088, 2048, "gated_gelu"), (40000, 1024, "f32"), (2056, 1088, "relu2")])
def test_matches_fp32(M, N, K, epi):
    a, w, res = _case(M, N, K, epi, pitch=64 if M == 17 else 0)
    bn = 0 if ops._stream_rule(M, N, K, epi, None) else 4001     # beyond the rule, but in the kernel's range
    got = ops.gemm(a, w, epi=epi, residual=res, bn=bn, w_ready=M % 2 == 0).float()
    want = ref.gemm(a.float(), w.float(), epi, res.float() if res is not None else None)
    # an output is rounded to bf16 once (2^-9); sums of K products in fp32 add K 2^-24 of their terms, below that
    scale = want.abs().clamp_min(1.0)
    assert ((got - want).abs() / scale).max().item() < (1e-4 if epi == "f32" else 2 ** -8)
    assert int(ops.gemm_status("cuda:0").item()) == 0


@pytest.mark.parametrize("splits", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("epi", ["store", "residual", "gated_silu"])
def test_shares_of_k_and_bias(splits, epi):
    a, w, res = _case(40, 1344, 1160, epi)   # 19 k-blocks: uneven shares
    bias = torch.randn(1344, device="cuda").bfloat16() if epi == "store" else None
    got = ops.gemm(a, w, epi=epi, residual=res, bias=bias, bn=4000 + splits).float()
    want = ref.gemm(a.float(), w.float(), epi, res.float() if res is not None else None, bias.float() if bias is not None else None)
    assert ((got - want).abs() / want.abs().clamp_min(1.0)).max().item() < 2 ** -8
    again = ops.gemm(a, w, epi=epi, residual=res, bias=bias, bn=4000 + splits).float()
    assert torch.equal(got, again)


@pytest.mark.parametrize("w_ready", [False, True])
def test_weights_written_by_the_kernel_before(w_ready):
    """Without w_ready the weights may come from the kernel queued just before, with it from the one before that.  One buffer: it holds NaN
    until a programmatic launch writes other values into it every time, so weights that are fetched too early show."""
    M, N, K = 8, 4096, 4096
    one = torch.ones(K, device="cuda", dtype=torch.bfloat16)
    w = torch.empty(N, K, device="cuda", dtype=torch.bfloat16)
    for seed in range(12):
        a, src, _ = _case(M, N, K, "store", seed)
        scaled = ops.rmsnorm(src, one, 1e-6)
        x = ops.rmsnorm(a, one, 1e-6) if w_ready else a
        want = x.float() @ scaled.float().t()
        w.fill_(float("nan"))
        torch.cuda.synchronize()
        ops.rmsnorm(src, one, 1e-6, out=w)             # a programmatic launch that writes the weights
        if w_ready:
            x = ops.rmsnorm(a, one, 1e-6)              # the kernel queued just before the GEMM
        got = ops.gemm(x, w, w_ready=w_ready).float()
        assert ((got - want).abs() / want.abs().clamp_min(1.0)).max().item() < 2 ** -7   # values of up to 300: one rounding to bf16
