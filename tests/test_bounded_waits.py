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
