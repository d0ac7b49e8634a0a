"""The cluster sampler against the definition: the filters' support, and the draw itself (the generator restated in numpy)."""
import numpy as np
import pytest
import torch

from lightllm_b200 import ops
from lightllm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _mix(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _keys(x, seed, step):
    """x_i - log(-log(u_i)): the arg-max over the kept tokens is the draw."""
    with np.errstate(over="ignore"):
        i = np.arange(len(x), dtype=np.uint64)
        h = _mix(np.uint64(seed) ^ _mix(np.uint64(step) * np.uint64(0x100000001B3) + i))
    u = ((h >> np.uint64(40)).astype(np.float64) + 0.5) / 16777216.0
    return x - np.log(-np.log(u))


@pytest.mark.parametrize("V", [4095, 4096, 4099, 32000, 128256, 151936, 393216, 393217])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_draws(V, dtype):
    B = 12
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = (torch.randn(B, V + 8, device="cuda", generator=g) * 3).to(dtype)[:, :V]
    temp = torch.linspace(0.2, 1.5, B, device="cuda")
    top_p = torch.tensor([1.0, 0.9, 0.5, 0.99, 1.0, 0.05] * 2, device="cuda")
    top_k = torch.tensor([0, -1, 5, 40, 1, 2000, V, 1, 2, 200, 50, 3], dtype=torch.int32, device="cuda")
    seeds = torch.arange(B, device="cuda") * 977 + 5
    steps = torch.arange(B, dtype=torch.int64, device="cuda") * 3
    ids, lp = ops.sample(logits, temp, top_p, top_k, seeds, steps)
    again, lp2 = ops.sample(logits, temp, top_p, top_k, seeds, steps)
    assert torch.equal(ids, again) and torch.equal(lp, lp2)
    for b in range(B):
        k = int(top_k[b])
        x = logits[b].float() / (1.0 if k == 1 else float(temp[b]))
        logp = torch.log_softmax(x.double(), -1)
        i = int(ids[b])
        # a log-probability is a difference of logits up to about 70 in fp32, and the fast exp / log: 1e-5 of that
        assert abs(float(lp[b]) - float(logp[i])) < 1e-3
        if k == 1:
            assert i == int(x.argmax())
            continue
        keep = ref.filtered_support(x, float(top_p[b]), k if k > 0 else V).cpu().numpy()
        key = _keys(x.double().cpu().numpy(), int(seeds[b]), int(steps[b]))
        best = np.where(keep, key, -np.inf).max()
        assert key[i] > best - 1e-3                      # the winner (or one within rounding of it) ...
        edge = x.cpu().numpy()[keep].min()
        assert float(x[i]) > edge - 1e-4                 # ... of the kept tokens


@pytest.mark.parametrize("V,pad", [(1, 0), (7, 0), (2049, 0), (4099, 5), (40000, 0), (128256, 8), (128257, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_greedy(V, pad, dtype):
    """The arg-max (the first of equal ones) and its log-probability, rows on any boundary, logits of -inf among them."""
    B = 5
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(B, V + pad, device="cuda", generator=g) * 4).to(dtype)[:, :V]
    x[1] = 0                       # all equal
    x[2, : V // 2] = float("-inf")
    x[3, V - 1] = 50
    x[4, : V - 1] = float("-inf")
    ids, lp = ops.sample(x)
    want = torch.stack([(r == r.max()).nonzero()[0, 0] for r in x])
    assert torch.equal(ids, want)
    ref_lp = torch.log_softmax(x.double(), -1).gather(1, want[:, None])[:, 0]
    assert (lp.double() - ref_lp).abs().max().item() < 1e-4   # fp32 sums of up to 1e5 positive terms, fast exp and log


@pytest.mark.parametrize("V", [100, 5000])
def test_a_row_of_nan(V):
    """A row without a single number has no token: the index says so, nothing is read there, and the other rows are drawn as they are alone."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(3, V, device="cuda", generator=g)
    args = [torch.full((3,), t, device="cuda") for t in (0.8, 0.9)] + [torch.full((3,), 20, dtype=torch.int32, device="cuda")] + \
        [torch.arange(3, device="cuda") + s for s in (5, 7)]
    want, want_lp = ops.sample(x, *args)
    x[1] = float("nan")
    ids, lp = ops.sample(x, *args)
    assert ids[1] == 0x7fffffff and lp[1].isnan()
    assert torch.equal(ids[::2], want[::2]) and torch.equal(lp[::2], want_lp[::2])
