"""What the framework's speed is judged by: passes of served models through the public engine API.

Three kinds of pass, on the model shapes that the benchmark and its serving configurations name (fewer layers, so that
several copies fit one GPU; every layer has its full width):

  decode    one step of `model.forward` for a running batch (captured graph, paged cache, per-step index tensors from
            pinned host memory) and the sampling of its tokens
  prefill   one prompt pass of `model.forward`: whole prompts, or chunks behind a cached prefix, lengths ragged
  generate  `LLM.generate`: admission, chunked prefill, decode and stop checks for a handful of prompts

Weights and caches come from the seed.  They keep what matters in served models: a residual stream of about 1 that
each layer changes by some tenths, attention scores and router logits with a spread of 2 to 3, and an output layer that
prefers two tokens, the first of them clearly (fixed successors of the last token, whose embedding is mixed into their
rows), so that the sampled tokens do not hang on the last bit.
"""
import hashlib
import math
import types

import numpy as np
import torch

BF, F8 = torch.bfloat16, torch.float8_e4m3fn

MODELS = {
    # Llama-3-8B shapes; 8 of 32 layers
    "llama3-8b": dict(model_type="llama", hidden_size=4096, num_hidden_layers=8, num_attention_heads=32,
                      num_key_value_heads=8, head_dim=128, intermediate_size=14336, vocab_size=128256, rms_norm_eps=1e-5,
                      rope_theta=5e5, eos_token_id=128001, torch_dtype="bfloat16"),
    # Llama-3-70B shapes; 2 of 80 layers
    "llama3-70b": dict(model_type="llama", hidden_size=8192, num_hidden_layers=2, num_attention_heads=64,
                       num_key_value_heads=8, head_dim=128, intermediate_size=28672, vocab_size=128256, rms_norm_eps=1e-5,
                       rope_theta=5e5, eos_token_id=128001, torch_dtype="bfloat16"),
    # Qwen3-30B-A3B shapes; 4 of 48 layers
    "qwen3-30b-a3b": dict(model_type="qwen3_moe", hidden_size=2048, num_hidden_layers=4, num_attention_heads=32,
                          num_key_value_heads=4, head_dim=128, intermediate_size=6144, moe_intermediate_size=768,
                          num_experts=128, num_experts_per_tok=8, norm_topk_prob=True, decoder_sparse_step=1,
                          mlp_only_layers=[], vocab_size=151936, rms_norm_eps=1e-6, rope_theta=1e6, eos_token_id=151645,
                          torch_dtype="bfloat16"),
    # DeepSeek-V3 shapes, e4m3 weights with 128 x 128 block scales; 2 of 61 layers (one dense, one of experts), 64 of
    # 256 routed experts: between the 32 that a GPU of eight holds and all of them
    "deepseek-v3": dict(model_type="deepseek_v3", hidden_size=7168, num_hidden_layers=2, num_attention_heads=128,
                        num_key_value_heads=128, q_lora_rank=1536, kv_lora_rank=512, qk_nope_head_dim=128,
                        qk_rope_head_dim=64, v_head_dim=128, intermediate_size=18432, moe_intermediate_size=2048,
                        n_routed_experts=64, n_shared_experts=1, num_experts_per_tok=8, n_group=8, topk_group=4,
                        first_k_dense_replace=1, moe_layer_freq=1, routed_scaling_factor=2.5, norm_topk_prob=True,
                        scoring_func="sigmoid", topk_method="noaux_tc", vocab_size=129280, rms_norm_eps=1e-6,
                        rope_theta=10000.0, eos_token_id=1, torch_dtype="bfloat16",
                        quantization_config={"quant_method": "fp8", "fmt": "e4m3", "activation_scheme": "dynamic",
                                             "weight_block_size": [128, 128]}),
}


def listed():
    def decode(name, model, batch, lo, hi, kv="bf16", quant="none", sampling="greedy"):
        return dict(name=name, kind="decode", model=model, batch=batch, ctx_lo=lo, ctx_hi=hi, kv=kv, quant=quant,
                    sampling=sampling)

    def prefill(name, model, batch, lo, hi, prefix, kv="bf16", quant="none"):
        return dict(name=name, kind="prefill", model=model, batch=batch, new_lo=lo, new_hi=hi, prefix=prefix, kv=kv,
                    quant=quant)

    return [
        # one user waiting for the next token: latency of the launches and of the weights' way through the chip
        decode("8b decode 1", "llama3-8b", 1, 700, 700),
        # a lightly loaded chat server: ragged contexts, temperature / top-p / top-k sampling
        decode("8b decode 24 sampled", "llama3-8b", 24, 200, 6000, sampling="random"),
        # the headline: 256 requests at once, 1024 tokens in, 256 out, somewhere in the output
        decode("8b decode 256", "llama3-8b", 256, 1025, 1280),
        # long documents over the 8-bit cache
        decode("8b decode 37 long fp8kv", "llama3-8b", 37, 3000, 12000, kv="fp8kv_sph"),
        # the headline's prompt pass: the largest that `batch_max_tokens` lets through
        prefill("8b prefill 16x1024", "llama3-8b", 16, 1024, 1024, 0),
        # what chunked prefill and the prefix cache make of mixed traffic: odd pieces behind cached prefixes
        prefill("8b prefill 6 ragged", "llama3-8b", 6, 37, 2900, 6000),
        # large dense model with weights quantised to fp8 at load
        decode("70b decode 64 fp8", "llama3-70b", 64, 130, 4096, quant="fp8w8a8-b128"),
        # experts: most of them have a few tokens each / hundreds each
        decode("moe decode 64", "qwen3-30b-a3b", 64, 2048, 2560),
        prefill("moe prefill 4x2048", "qwen3-30b-a3b", 4, 2048, 2048, 0),
        # latent attention, fp8 experts
        decode("deepseek decode 96", "deepseek-v3", 96, 1025, 2048),
        prefill("deepseek prefill 7 ragged", "deepseek-v3", 7, 300, 1500, 1000),
        # the whole engine on a burst of chat prompts
        dict(name="8b generate 24", kind="generate", model="llama3-8b", batch=24, new_lo=17, new_hi=900, out=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "generate"])
    if kind == "generate":
        return dict(kind=kind, model="llama3-8b", batch=_log(rng, 4, 24), new_lo=_log(rng, 8, 60), new_hi=_log(rng, 100, 900),
                    out=rng.randint(8, 24))
    model = rng.choice(list(MODELS))
    llama = model.startswith("llama")
    kv = rng.choice(["bf16", "bf16", "int8kv", "fp8kv_sph"]) if llama else "bf16"
    quant = rng.choice(["none", "fp8w8a8-b128"]) if model == "llama3-70b" else "none"
    if kind == "decode":
        batch = _log(rng, 1, 256 if model == "llama3-8b" else 128)
        hi = _log(rng, 100, min(12000, 330000 // batch))
        return dict(kind=kind, model=model, batch=batch, ctx_lo=rng.randint(max(2, hi // 8), hi), ctx_hi=hi, kv=kv, quant=quant,
                    sampling=rng.choice(["greedy", "greedy", "random"]))
    batch = _log(rng, 1, 12)
    hi = _log(rng, 40, min(4000, (12000 if model == "llama3-8b" else 6000) // batch))
    return dict(kind=kind, model=model, batch=batch, new_lo=rng.randint(max(1, hi // 8), hi), new_hi=hi,
                prefix=rng.choice([0, 0, _log(rng, 16, 6000 if model == "llama3-8b" else 1500)]), kv=kv, quant=quant)


# ---------------------------------------------------------------------------------------------------------- inputs
def _gen(seed, name, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    return g


def _normal(seed, name, shape, std=1.0, dtype=BF):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=_gen(seed, name))


def _shapes(c):
    """Checkpoint names -> (shape, standard deviation; None: a norm's weight)."""
    H, V, n = c["hidden_size"], c["vocab_size"], c["num_hidden_layers"]
    ffn = 0.35 if "quantization_config" in c else 0.6   # fp8 activations: noise of some percent in what a layer adds
    s = {"model.embed_tokens.weight": ((V, H), 1.0), "model.norm.weight": ((H,), None), "lm_head.weight": ((V, H), 0.2 / H ** 0.5)}

    def lin(name, out, inp, gain):
        s[name] = ((out, inp), gain / inp ** 0.5)

    def mlp(p, inter, gain):
        lin(p + "gate_proj.weight", inter, H, 1.0)
        lin(p + "up_proj.weight", inter, H, 1.0)
        lin(p + "down_proj.weight", H, inter, gain)

    for i in range(n):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        s[p + "input_layernorm.weight"] = s[p + "post_attention_layernorm.weight"] = ((H,), None)
        hq = c["num_attention_heads"]
        if "kv_lora_rank" in c:
            nope, rope, dv, kvl, ql = (c[k] for k in ("qk_nope_head_dim", "qk_rope_head_dim", "v_head_dim", "kv_lora_rank",
                                                      "q_lora_rank"))
            lin(a + "q_a_proj.weight", ql, H, 1.0)
            s[a + "q_a_layernorm.weight"], s[a + "kv_a_layernorm.weight"] = ((ql,), None), ((kvl,), None)
            lin(a + "q_b_proj.weight", hq * (nope + rope), ql, 1.6)
            lin(a + "kv_a_proj_with_mqa.weight", kvl + rope, H, 1.0)
            lin(a + "kv_b_proj.weight", hq * (nope + dv), kvl, 1.2)
            lin(a + "o_proj.weight", H, hq * dv, 0.35)
        else:
            D, hkv = c["head_dim"], c["num_key_value_heads"]
            lin(a + "q_proj.weight", hq * D, H, 1.4)
            lin(a + "k_proj.weight", hkv * D, H, 1.4)
            lin(a + "v_proj.weight", hkv * D, H, 1.0)
            lin(a + "o_proj.weight", H, hq * D, 0.6)
            if c["model_type"].startswith("qwen3"):
                s[a + "q_norm.weight"] = s[a + "k_norm.weight"] = ((D,), None)
        E = c.get("num_experts") or c.get("n_routed_experts")
        if E and i >= c.get("first_k_dense_replace", 0):
            lin(p + "mlp.gate.weight", E, H, 3.0 if "num_experts" in c else 1.0)
            if c.get("topk_method") == "noaux_tc":
                s[p + "mlp.gate.e_score_correction_bias"] = ((E,), 0.05)
            for e in range(E):
                mlp(p + f"mlp.experts.{e}.", c["moe_intermediate_size"], ffn if "num_experts" in c else 0.15)
            if c.get("n_shared_experts"):
                mlp(p + "mlp.shared_experts.", c["moe_intermediate_size"] * c["n_shared_experts"], ffn)
        else:
            mlp(p + "mlp.", c["intermediate_size"], ffn)
    return s


class Checkpoint:
    """The tensors of a checkpoint, each made from the seed and its name when it is asked for."""

    def __init__(self, cfg, seed):
        self.cfg, self.seed, self.spec = cfg, seed, _shapes(cfg)
        self.fp8 = "quantization_config" in cfg

    def _is_fp8(self, n):
        return self.fp8 and n.endswith("proj.weight")      # kv_a_proj_with_mqa stays in 16 bits

    def has(self, n):
        return n in self.spec or (n.endswith("_scale_inv") and n[:-len("_scale_inv")] in self.spec and
                                  self._is_fp8(n[:-len("_scale_inv")]))

    def names(self):
        return list(self.spec) + [n + "_scale_inv" for n in self.spec if self._is_fp8(n)]

    def shape(self, n):
        if n.endswith("_scale_inv"):
            r, c = self.spec[n[:-len("_scale_inv")]][0]
            return (-(-r // 128), -(-c // 128))
        return self.spec[n][0]

    def full(self, n):
        if n.endswith("_scale_inv"):
            std = self.spec[n[:-len("_scale_inv")]][1]
            return (torch.rand(self.shape(n), generator=_gen(self.seed, n), device="cuda") * 0.6 + 0.7) * (std / 96.0)
        shape, std = self.spec[n]
        if std is None:
            return (1.0 + 0.1 * _normal(self.seed, n, shape, dtype=torch.float32)).to(BF)
        if n.endswith("correction_bias"):
            return _normal(self.seed, n, shape, std, torch.float32)
        if self._is_fp8(n):
            return _normal(self.seed, n, shape, 96.0).clamp_(-448, 448).to(F8)
        w = _normal(self.seed, n, shape, std)
        if n == "lm_head.weight":
            V, H = shape
            v, emb = torch.arange(V, device="cuda"), self.full("model.embed_tokens.weight")
            w[next_token(v, V)] += emb * (20.0 / H)
            w[second_token(v, V)] += emb * (14.0 / H)
        return w

    def get(self, n, dim=None, start=0, end=None):
        t = self.full(n)
        if dim is not None:
            t = t.narrow(dim, start, (t.shape[dim] if end is None else end) - start)
        return t

    def exact(self, n):
        """The tensor in 64 bits, block scales applied."""
        t = self.full(n).double()
        if self._is_fp8(n):
            s = self.full(n + "_scale_inv").double().repeat_interleave(128, 0)[:t.shape[0]]
            t *= s.repeat_interleave(128, 1)[:, :t.shape[1]]
        return t


def next_token(v, vocab):
    return (v * 31 + 7) % vocab   # a permutation: 31 divides none of the vocabulary sizes, nor does 37


def second_token(v, vocab):
    return (v * 37 + 11) % vocab


def _lengths(case, seed):
    """(cached, new) tokens of the requests: lengths from lo to hi, hi among them, spread over their logarithm.  The set of
    them belongs to the case; the seed only says which request has which."""
    B = case["batch"]
    lo, hi = (case["ctx_lo"], case["ctx_hi"]) if case["kind"] == "decode" else (case["new_lo"], case["new_hi"])
    u = torch.rand(B, generator=_gen(0, f"lengths {B} {lo} {hi}", "cpu"), dtype=torch.float64)
    got = (math.log(lo) + u * (math.log(hi) - math.log(lo))).exp().round().long().clamp(lo, hi)
    got[0] = hi
    if case["kind"] == "decode":
        ready, new = got - 1, torch.ones_like(got)
    else:
        prefix = case.get("prefix", 0)
        u = torch.rand(B, generator=_gen(0, f"prefixes {B} {prefix}", "cpu"))
        ready, new = (u * u * (prefix + 1)).long() if prefix else torch.zeros_like(got), got
    order = torch.randperm(B, generator=_gen(seed, "who", "cpu"))
    return ready[order], new[order]


def _plan(case, seed):
    """Tokens and pool slots of a pass: ready (cached) and new tokens per request, slots of all positions.

    Cached tokens lie in runs, as prompts leave them, with a decoded tail whose slots alternate between the requests;
    the pass's own slots follow one another."""
    B = case["batch"]
    ready, new = _lengths(case, seed)
    tail = torch.minimum(ready // 4, torch.tensor(200)) if case["kind"] == "decode" else torch.zeros_like(ready)
    slots, at = [None] * B, 0
    for b in torch.randperm(B, generator=_gen(seed, "order", "cpu")).tolist():
        n = int(ready[b] - tail[b])
        slots[b] = [torch.arange(at, at + n)]
        at += n
    for t in range(int(tail.max())):
        live = (tail > t).nonzero().view(-1).tolist()
        for k, b in enumerate(live):
            slots[b].append(torch.tensor([at + k]))
        at += len(live)
    first_new = at
    for b in range(B):
        n = int(new[b])
        slots[b] = torch.cat(slots[b] + [torch.arange(at, at + n)])
        at += n
    vocab = MODELS[case["model"]]["vocab_size"]
    ids = torch.randint(1000, vocab - 1000, (int(new.sum()),), generator=_gen(seed, "ids", "cpu"))
    return types.SimpleNamespace(B=B, ready=ready, new=new, slots=slots, first_new=first_new, total=at, ids=ids,
                                 seq=ready + new)


def _fill_pool(buf, case, seed):
    """Cached keys and values (layer by layer), as an earlier pass would have left them."""
    c = MODELS[case["model"]]
    for i in range(c["num_hidden_layers"]):
        row = buf[i].shape[1:]
        n = buf[i].shape[0]
        v = _normal(seed, f"pool{i}", (n, row[0], c["head_dim"] if "head_dim" in c else row[1]))
        if "head_dim" in c:
            v[:, : row[0] // 2] *= 1.4
        if case["kv"] == "fp8kv_sph":                 # rows in e4m3, scale 1
            buf[i].view(F8).copy_(v)
        elif case["kv"] == "int8kv":                  # 128 values and their fp32 scale in 16 more bytes
            s = v.abs().amax(-1, keepdim=True).float() / 127
            buf[i][..., :128] = (v / s).round().to(torch.int8)
            buf[i][..., 128:132] = s.contiguous().view(torch.int8)
        else:
            buf[i].copy_(v)
        del v


def _pool_rows(rows, case):
    """Rows of a pool as _fill_pool wrote them -> 64 bits."""
    if case["kv"] == "fp8kv_sph":
        return rows.view(F8).double()
    if case["kv"] == "int8kv":
        return rows[..., :128].double() * rows[..., 128:132].contiguous().view(torch.float32).double()
    return rows.double()


def _pool_shape(case, slots):
    c = MODELS[case["model"]]
    n = c["num_hidden_layers"]
    if "kv_lora_rank" in c:
        return (n, slots, 1, c["kv_lora_rank"] + c["qk_rope_head_dim"]), BF
    if case["kv"] == "int8kv":
        return (n, slots, 2 * c["num_key_value_heads"], c["head_dim"] + 16), torch.int8
    return (n, slots, 2 * c["num_key_value_heads"], c["head_dim"]), torch.uint8 if case["kv"] == "fp8kv_sph" else BF


def _sampling(case, seed):
    if case.get("sampling") != "random":
        return None
    B = case["batch"]
    g = _gen(seed, "sampling", "cpu")
    return dict(temperature=torch.rand(B, generator=g) * 0.3 + 0.1, top_p=torch.rand(B, generator=g) * 0.4 + 0.6,
                top_k=torch.randint(2, 200, (B,), generator=g, dtype=torch.int32),
                seeds=torch.randint(1 << 40, (B,), generator=g), steps=torch.arange(B, dtype=torch.int32))


# ---------------------------------------------------------------------------------------------------------- the passes
def _llm(case, seed, **kw):
    from lightllm_b200.engine.llm import LLM
    from lightllm_b200.parallel import dist as pdist

    if pdist.state().device.type != "cuda":
        pdist.init_distributed(1, 0, device=torch.device("cuda", 0))
    cfg = dict(MODELS[case["model"]])
    if case.get("kv", "bf16") != "bf16":
        kw["kv_type"] = case["kv"]
    if case.get("quant", "none") != "none":
        kw["quant_type"] = case["quant"]
    return LLM(config=cfg, weight_source=Checkpoint(cfg, seed), **kw)


def _prompts(case, seed):
    n = _lengths(case, seed)[1].tolist()
    vocab = MODELS[case["model"]]["vocab_size"]
    ids = torch.randint(1000, vocab - 1000, (sum(n),), generator=_gen(seed, "ids", "cpu"))
    return [t.tolist() for t in ids.split(n)]


def prepare(case, seed):
    s = types.SimpleNamespace(kind=case["kind"])
    if case["kind"] == "generate":
        total = case["new_hi"] + case["out"]
        s.llm = _llm(case, seed, max_total_token_num=case["batch"] * (total + 8) + 4096, running_max_req_size=32,
                     max_req_total_len=total + 8, batch_max_tokens=8192, disable_dynamic_prompt_cache=True,
                     graph_max_batch_size=case["batch"])
        s.llm.warmup()
        s.prompts, s.params = _prompts(case, seed), {"max_new_tokens": case["out"], "ignore_eos": True}
        return s
    p = _plan(case, seed)
    longest = int(p.seq.max())
    T = int(p.new.sum())
    s.llm = _llm(case, seed, max_total_token_num=p.total, running_max_req_size=p.B, max_req_total_len=longest + 256,
                 batch_max_tokens=max(T, 2048), graph_max_batch_size=p.B, disable_dynamic_prompt_cache=True)
    m = s.model = s.llm.model
    mm, rm = m.mem_manager, m.req_manager
    _fill_pool(mm.kv_buffer, case, seed)
    for b in range(p.B):
        n = int(p.ready[b])
        rm.req_to_token_indexs[b, :n] = p.slots[b][:n].to(rm.req_to_token_indexs)
    new = mm.kv_buffer[:, p.first_new:p.total]
    s.new_rows = new.view(F8) if case["kv"] == "fp8kv_sph" else new
    s.int8 = case["kv"] == "int8kv"
    pin = lambda t, dt=torch.int32: t.to(dt).contiguous().pin_memory()  # noqa: E731
    s.args = dict(batch_size=p.B, total_token_num=int(p.seq.sum()), max_kv_len=longest,
                  is_prefill=case["kind"] == "prefill", b_req_idx=pin(torch.arange(p.B)), b_seq_len=pin(p.seq),
                  mem_indexes=pin(torch.arange(p.first_new, p.total)))
    s.sampling = {}
    if case["kind"] == "prefill":
        s.args.update(input_ids=pin(p.ids, torch.int64), b_ready_cache_len=pin(p.ready), b_q_len=pin(p.new),
                      max_q_len=int(p.new.max()))
    else:
        rm.req_to_next_token_ids[:p.B, 0] = p.ids.to(rm.req_to_next_token_ids)
        s.llm.warmup([p.B])
        s.sampling = {k: v.cuda() for k, v in (_sampling(case, seed) or {}).items()}
    return s


def run(state):
    """A pass: logits, tokens, their log probabilities and the cache rows that it wrote."""
    if state.kind == "generate":
        outs = state.llm.generate(state.prompts, state.params)
        return {"tokens": np.array([o["token_ids"] for o in outs]),
                "logprobs": np.array([o["logprobs"] for o in outs], dtype=np.float32)}
    from lightllm_b200 import ops
    from lightllm_b200.common.infer_state import ModelInput

    out = state.model.forward(ModelInput(**state.args))
    tokens, logprobs = ops.sample(out.logits_any, **state.sampling)
    got = {"logits": out.logits, "tokens": tokens}
    if not state.sampling:   # at a low temperature they are rounding errors of the winner's probability of almost 1
        got["logprobs"] = logprobs
    if not state.int8:       # bytes whose last bit may go either way: the step's own attention has read those rows
        got["rows"] = state.new_rows
    return got


# ---------------------------------------------------------------------------------------------------------- the work
def work(case):
    """Bytes: weights that the pass needs once, cached rows read, new rows, logits written.  Operations: matrix products
    and the visible part of attention."""
    c = MODELS[case["model"]]
    H, V, n, hq = c["hidden_size"], c["vocab_size"], c["num_hidden_layers"], c["num_attention_heads"]
    wb = 1 if "quantization_config" in c or case.get("quant", "none") != "none" else 2
    if case["kind"] == "generate":
        new = _lengths(case, 0)[1].double()
        seqs, out_rows, passes = [(torch.zeros_like(new), new)], case["batch"], case["out"]
        for t in range(1, case["out"]):
            seqs.append((new + t - 1, torch.ones_like(new)))
            out_rows += case["batch"]
    else:
        ready, new = _lengths(case, 0)
        seqs, out_rows, passes = [(ready.double(), new.double())], case["batch"], 1
    E = c.get("num_experts") or c.get("n_routed_experts") or 0
    k = c.get("num_experts_per_tok", 0)
    flops = bytes_ = 0.0
    for ready, new in seqs:
        T = float(new.sum())
        pairs = float((new * ready + new * (new + 1) / 2).sum())   # (query, visible key)
        per_tok = per_pass = 0.0
        if "kv_lora_rank" in c:
            nope, rope, dv, kvl, ql = (c[x] for x in ("qk_nope_head_dim", "qk_rope_head_dim", "v_head_dim", "kv_lora_rank",
                                                      "q_lora_rank"))
            attn = H * (ql + kvl + rope) + ql * hq * (nope + rope) + kvl * hq * (nope + dv) + hq * dv * H
            absorbed = T == len(new)
            a_flops = 2 * hq * pairs * ((2 * kvl + rope) if absorbed else (nope + rope + dv))
            row = 2.0 * (kvl + rope)
        else:
            D, hkv = c["head_dim"], c["num_key_value_heads"]
            attn = H * (hq + 2 * hkv) * D + hq * D * H
            a_flops = 4 * hq * D * pairs
            row = 2 * hkv * D * {"bf16": 2.0, "fp8kv_sph": 1.0, "int8kv": 1.03}[case.get("kv", "bf16")]
        for i in range(n):
            per_tok += attn
            per_pass += attn
            if E and i >= c.get("first_k_dense_replace", 0):
                one = 3 * H * c["moe_intermediate_size"]
                shared = one * c.get("n_shared_experts", 0)
                per_tok += k * one + shared + E * H
                per_pass += E * (1 - (1 - k / E) ** T) * one + shared + E * H
            else:
                per_tok += 3 * H * c["intermediate_size"]
                per_pass += 3 * H * c["intermediate_size"]
        flops += 2 * T * per_tok + n * a_flops
        bytes_ += per_pass * wb + n * row * float((ready + 2 * new).sum()) + T * H * 2
    flops += 2.0 * out_rows * H * V
    bytes_ += passes * H * V * 2.0 + out_rows * V * 4.0
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Logits of the 16-bit passes end about 0.01 from the 64-bit ones, those with fp8 activations 0.02 to 0.04; another order
    of the sums, or another place for a rounding, moves them by about as much again.  Tokens are the same."""
    return {"rel": 0.03, "max": 0.6, "differ": 0.0}


# ---------------------------------------------------------------------------------------------------------- in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, theta, pairs):
    """x [T, heads, d] turned by its position: pairs of neighbours, or of halves."""
    d = x.shape[-1]
    ang = pos.double()[:, None] / theta ** (torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = (x[..., 0::2], x[..., 1::2]) if pairs else (x[..., : d // 2], x[..., d // 2:])
    return torch.cat([a * c - b * s, b * c + a * s], -1)   # halves in either case


def _attend(q, k, v, ready, scale):
    """q [n, h, d] behind `ready` positions, k [L, hk, d], v [L, hk, dv] -> [n, h, dv]."""
    n, h, _ = q.shape
    L, hk = k.shape[0], k.shape[1]
    g = h // hk
    out = torch.empty(n, h, v.shape[-1], dtype=torch.float64, device=q.device)
    seen = torch.arange(L, device=q.device)[None] <= torch.arange(n, device=q.device)[:, None] + ready
    step = max(1, (1 << 27) // max(1, n * L * g))
    for a in range(0, hk, step):
        e = min(hk, a + step)
        qq = q[:, a * g:e * g].reshape(n, e - a, g, -1)
        s = torch.einsum("nkgd,lkd->kgnl", qq, k[:, a:e]) * scale
        s.masked_fill_(~seen, float("-inf"))
        o = torch.einsum("kgnl,lkd->nkgd", torch.softmax(s, -1), v[:, a:e])
        out[:, a * g:e * g] = o.reshape(n, (e - a) * g, -1)
    return out


def _mlp(x, w, p):
    return (torch.nn.functional.silu(x @ w.exact(p + "gate_proj.weight").t()) *
            (x @ w.exact(p + "up_proj.weight").t())) @ w.exact(p + "down_proj.weight").t()


def _experts(x, c, w, p):
    E, k = c.get("num_experts") or c["n_routed_experts"], c["num_experts_per_tok"]
    logits = x @ w.exact(p + "gate.weight").t()
    if "num_experts" in c:
        val, idx = logits.softmax(-1).topk(k, -1)
        val = val / val.sum(-1, keepdim=True)
    else:
        score = logits.sigmoid()
        pick = (score + w.exact(p + "gate.e_score_correction_bias")).view(len(x), c["n_group"], -1)
        best = pick.topk(2, -1).values.sum(-1).topk(c["topk_group"], -1).indices
        keep = torch.zeros(pick.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, best, True)
        idx = pick.masked_fill(~keep[..., None], float("-inf")).view(len(x), E).topk(k, -1).indices
        val = score.gather(1, idx)
        val = val / val.sum(-1, keepdim=True) * c["routed_scaling_factor"]
    out = torch.zeros_like(x)
    for e in range(E):
        t, j = (idx == e).nonzero(as_tuple=True)
        if len(t):
            out.index_add_(0, t, _mlp(x[t], w, p + f"experts.{e}.") * val[t, j, None])
    if c.get("n_shared_experts"):
        out += _mlp(x, w, p + "shared_experts.")
    return out


def _forward(c, w, ids, ready, new, cached):
    """The model on new tokens `ids` behind cached rows: (last hidden rows, normed; rows that were added per layer)."""
    eps, hq = c["rms_norm_eps"], c["num_attention_heads"]
    pos = torch.cat([torch.arange(r, r + n) for r, n in zip(ready, new)]).cuda()
    x = w.full("model.embed_tokens.weight")[ids.cuda()].double()
    rows = []
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        h = _rms(x, w.exact(p + "input_layernorm.weight"), eps)
        if "kv_lora_rank" in c:
            nope, rope, dv, kvl = (c[t] for t in ("qk_nope_head_dim", "qk_rope_head_dim", "v_head_dim", "kv_lora_rank"))
            q = _rms(h @ w.exact(a + "q_a_proj.weight").t(), w.exact(a + "q_a_layernorm.weight"), eps)
            q = (q @ w.exact(a + "q_b_proj.weight").t()).view(-1, hq, nope + rope)
            q = torch.cat([q[..., :nope], _rotate(q[..., nope:], pos, c["rope_theta"], True)], -1)
            kv = h @ w.exact(a + "kv_a_proj_with_mqa.weight").t()
            lat = _rms(kv[:, :kvl], w.exact(a + "kv_a_layernorm.weight"), eps)
            row = torch.cat([lat, _rotate(kv[:, None, kvl:], pos, c["rope_theta"], True)[:, 0]], -1)[:, None]
            up = w.exact(a + "kv_b_proj.weight").view(hq, nope + dv, kvl)
            scale = (nope + rope) ** -0.5
        else:
            D, hkv = c["head_dim"], c["num_key_value_heads"]
            q, k, v = ((h @ w.exact(a + t + "_proj.weight").t()).view(len(h), -1, D) for t in "qkv")
            if w.has(a + "q_norm.weight"):
                q, k = _rms(q, w.exact(a + "q_norm.weight"), eps), _rms(k, w.exact(a + "k_norm.weight"), eps)
            q, k = _rotate(q, pos, c["rope_theta"], False), _rotate(k, pos, c["rope_theta"], False)
            row = torch.cat([k, v], 1)
            scale = D ** -0.5
        o, at = [], 0
        for b, n in enumerate(new):
            all_rows = torch.cat([cached(i, b), row[at:at + n]])
            if "kv_lora_rank" in c:
                kvb = torch.einsum("lr,hdr->lhd", all_rows[:, 0, :kvl], up)
                kk = torch.cat([kvb[..., :nope], all_rows[:, :, kvl:].expand(-1, hq, -1)], -1)
                vv = kvb[..., nope:]
            else:
                kk, vv = all_rows[:, :hkv], all_rows[:, hkv:]
            o.append(_attend(q[at:at + n], kk, vv, ready[b], scale).reshape(n, -1))
            at += n
        rows.append(row)
        x = x + torch.cat(o) @ w.exact(a + "o_proj.weight").t()
        h = _rms(x, w.exact(p + "post_attention_layernorm.weight"), eps)
        x = x + (_experts(h, c, w, p + "mlp.") if w.has(p + "mlp.gate.weight") else _mlp(h, w, p + "mlp."))
    return _rms(x, w.exact("model.norm.weight"), eps), torch.stack(rows)


def _logits(h, w):
    head = w.full("lm_head.weight")
    return torch.cat([h @ part.double().t() for part in head.split(16384)], -1)


def exact(case, seed):
    c = MODELS[case["model"]]
    w = Checkpoint(c, seed)
    if case["kind"] == "generate":   # the tokens follow from the prompts: score them in one pass
        seqs, V = _prompts(case, seed), c["vocab_size"]
        for s in seqs:
            for _ in range(case["out"] - 1):
                s.append(next_token(s[-1], V))
        lens = [len(s) for s in seqs]
        none = torch.zeros(0, 2 * c["num_key_value_heads"], c["head_dim"], dtype=torch.float64, device="cuda")
        h, _ = _forward(c, w, torch.tensor(sum(seqs, [])), [0] * len(seqs), lens, lambda i, b: none)
        got, end = [], 0
        for s, n in zip(seqs, lens):
            end += n
            want = torch.tensor([next_token(t, V) for t in s[-case["out"]:]], device="cuda")
            lp = _logits(h[end - case["out"]:end], w).log_softmax(-1)
            got.append(lp.gather(1, want[:, None])[:, 0])
        return {"tokens": None, "logprobs": torch.stack(got)}
    p = _plan(case, seed)
    shape, dtype = _pool_shape(case, p.total + 1)
    pool = torch.zeros(shape, dtype=dtype, device="cuda")
    _fill_pool(pool, case, seed)
    cached = lambda i, b: _pool_rows(pool[i][p.slots[b][: int(p.ready[b])].cuda()], case)  # noqa: E731
    h, rows = _forward(c, w, p.ids, p.ready.tolist(), p.new.tolist(), cached)
    logits = _logits(h[(p.new.cumsum(0) - 1).cuda()], w)
    out = {"logits": logits, "tokens": None}
    if case.get("sampling") != "random":
        out["logprobs"] = logits.log_softmax(-1).amax(-1)
    if case["kv"] != "int8kv":
        out["rows"] = rows
    return out
