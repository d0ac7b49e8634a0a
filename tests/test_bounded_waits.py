"""Bounded waits in the kernels' issuing threads: a wait that ran out (mbar_wait returns false) ends the issuing.  An MMA issued all the same
would read stages whose copies are still in flight.  A wait cannot be made to run out in these kernels without breaking them, so the
sources are read."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "lightllm_b200" / "csrc"


@pytest.mark.parametrize("name", ["gemm_stream", "attention_fa", "mla_decode"])
def test_issuing_threads_heed_their_waits(name):
    text = re.sub(r"//[^\n]*", lambda m: m.group() if "MMA issuer" in m.group() else "", (CSRC / f"{name}.cu").read_text())
    part = text[text.index("MMA issuer"):]
    part = part[: part.index("__syncwarp();")]
    waits = re.findall(r"([^;{}]*)\bmbar_wait\(", part)
    assert waits and all(re.search(r"(if \(|return|&&|\|\||=)[^;]*$", w) for w in waits), waits


def test_prompt_attention_reports_to_the_shared_word(monkeypatch):
    """The codes of prompt attention arrive where those of the GEMMs do (on the CPU: the pointers that its launches get)."""
    import torch

    from lightllm_b200 import ops
    from lightllm_b200.ops import mla

    calls = {}

    class Fake:
        def __getattr__(self, name):
            return lambda *a: calls.setdefault(name, a) and 0

    word, i, z = torch.zeros(1, dtype=torch.int32), lambda *x: torch.tensor(x, dtype=torch.int32), lambda *s: torch.zeros(s, dtype=torch.bfloat16)
    for m in (ops, mla):
        monkeypatch.setattr(m, "kernels", Fake)
        monkeypatch.setattr(m, "gemm_status", lambda device: word)
        monkeypatch.setattr(m, "stream", lambda: None)
    monkeypatch.setattr(ops, "_is_cuda", lambda t: True)
    ops.gqa_prefill(z(4, 256), z(8, 4, 128), i(*range(8)).view(1, 8), i(0), i(0, 4), i(0), 2, 2, 128, 4)
    mla.latent_prefill(z(4, 384), z(4, 512), z(4, 576), 512, 128, 2, 192, 128, i(0, 4), i(0), mla.KeyRange(i(0), i(4), 0, "cpu"), 4, 0.1, z(4, 256))
    for name in ("llb_gqa_prefill_fa", "llb_latent_prefill_fa"):
        assert any(getattr(a, "value", None) == word.data_ptr() for a in calls[name]), name
