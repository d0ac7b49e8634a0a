"""Tuned-config store (nearest run key, user file shadows the shipped one) and the candidate benchmark split over
the ranks of a gloo group."""
import json
import os
import socket

import torch
import torch.multiprocessing as mp

from lightllm_b200.utils import autotuner as at


def test_store_lookup_and_shadowing(tmp_path, monkeypatch):
    shipped = tmp_path / "pkg"
    monkeypatch.setattr(at, "PKG_DIR", shipped)
    (shipped / "devX").mkdir(parents=True)
    (shipped / "devX" / "gemm_bf16.json").write_text(json.dumps(
        {"N=4096,K=4096,epi=store": {"16": {"bn": 64}, "256": {"bn": 1012}}}))
    st = at.KernelConfigStore(device="devX", user_dir=str(tmp_path / "user"))
    key = at.gemm_static_key(4096, 4096, "store")
    assert st.lookup("gemm_bf16", key, 1)["bn"] == 64 and st.lookup("gemm_bf16", key, 100)["bn"] == 64
    assert st.lookup("gemm_bf16", key, 136)["bn"] == 1012 and st.lookup("gemm_bf16", key, 4000)["bn"] == 1012
    assert st.lookup("gemm_bf16", "N=1,K=1,epi=store", 8) is None
    st.store("gemm_bf16", key, 16, {"bn": 128})          # the user's entry shadows the shipped one
    st.store("gemm_bf16", key, 64, {"bn": 1111})
    st2 = at.KernelConfigStore(device="devX", user_dir=str(tmp_path / "user"))
    assert st2.lookup("gemm_bf16", key, 16)["bn"] == 128 and st2.lookup("gemm_bf16", key, 70)["bn"] == 1111
    assert st2.has("gemm_bf16", key, 64) and not st2.has("gemm_bf16", key, 65)
    at.reset_store(st2)
    try:
        assert at.gemm_lookup(16, 4096, 4096, "store") == 128 and at.gemm_lookup(16, 8, 8, "store") == 0
    finally:
        at.reset_store(None)
    best, scored = at.tune([{"bn": 1}, {"bn": 2}, {"bn": 3}], lambda c: {1: 5.0, 2: 1.0, 3: 9.0}[c["bn"]])
    assert best == {"bn": 2} and [c["bn"] for _, c in scored] == [2, 1, 3]

    def failing(c):
        if c["bn"] == 2:
            raise RuntimeError("unsupported variant")
        return float(c["bn"])

    assert at.tune([{"bn": 1}, {"bn": 2}, {"bn": 3}], failing)[0] == {"bn": 1}


def _rank(rank, world, port, out):
    import torch.distributed as dist

    os.environ["MASTER_ADDR"], os.environ["MASTER_PORT"] = "127.0.0.1", str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    seen = []

    def bench(c):
        seen.append(c["bn"])
        return abs(c["bn"] - 7) + 0.5

    best, scored = at.tune([{"bn": b} for b in range(12)], bench, group=dist.group.WORLD)
    torch.save({"best": best, "seen": seen, "n": len(scored)}, os.path.join(out, f"r{rank}.pt"))
    dist.destroy_process_group()


def test_candidates_are_split_across_ranks(tmp_path):
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    port = s.getsockname()[1]
    s.close()
    mp.spawn(_rank, args=(2, port, str(tmp_path)), nprocs=2, join=True)
    a, b = torch.load(tmp_path / "r0.pt"), torch.load(tmp_path / "r1.pt")
    assert a["best"] == b["best"] == {"bn": 7} and a["n"] == b["n"] == 12
    assert sorted(a["seen"] + b["seen"]) == list(range(12)) and not set(a["seen"]) & set(b["seen"])


def test_few_token_gemm_and_stored_variants(tmp_path, monkeypatch):
    """Few tokens: a stored variant of the tile kernels counts if it was timed against the few-token kernel; a push to tensor-parallel peers,
    which only the tile kernels make, gets the best of those."""
    from lightllm_b200 import ops

    N, K, armed, calls = 4096, 4096, [0], []

    class Fake:
        def llb_gemm_push_armed(self):
            return armed[0]

        def llb_gemm_stream(self, *a):
            calls.append(("few", a[12].value))
            return 0

        def llb_gemm_bf16(self, *a):
            calls.append(("tile", a[12].value))
            return 0

    word = torch.zeros(1, dtype=torch.int32)
    for name, value in (("kernels", Fake), ("gemm_status", lambda d: word), ("stream", lambda: None), ("_is_cuda", lambda t: True),
                        ("_stream_k_scratch", lambda d: (word.float(), word))):
        monkeypatch.setattr(ops, name, value)
    monkeypatch.setattr(at, "PKG_DIR", tmp_path / "pkg")
    st = at.KernelConfigStore(device="devX", user_dir=str(tmp_path / "user"))
    key = at.gemm_static_key(N, K, "store")
    for M, cfg in ((1, {"bn": 2000}), (16, {"bn": 2002, "few": 1}), (32, {"bn": 4003, "few": 1, "tile": 2004}), (64, {"bn": 0, "few": 1, "tile": 1012})):
        st.store("gemm_bf16", key, M, cfg, save=False)
    at.reset_store(st)
    w = torch.zeros(N, K, dtype=torch.bfloat16)
    try:
        def route(M, push=0):
            armed[0] = push
            ops.gemm(torch.zeros(M, K, dtype=torch.bfloat16), w)
            return calls.pop()

        assert [route(M) for M in (1, 16, 32, 64)] == [("few", 0), ("tile", 2002), ("few", 3), ("few", 0)]
        assert [route(M, push=2) for M in (1, 16, 32, 64)] == [("tile", 2000), ("tile", 2002), ("tile", 2004), ("tile", 1012)]
    finally:
        at.reset_store(None)


def test_shipped_table_keeps_the_variants_of_few_tokens():
    """A row-parallel projection of a tensor-parallel rank is pushed to its peers by the tile kernels with 1 to 8 tokens too: the variants
    tuned at those sizes are there, not the nearest one of 128 tokens."""
    table = json.loads((at.PKG_DIR / "NVIDIA_B200" / "gemm_bf16.json").read_text())
    for N, K in ((4096, 1024), (4096, 1792), (4096, 2048), (4096, 3584), (4096, 7168), (8192, 1024), (8192, 3584)):
        assert {"1", "8", "16", "32", "64", "128"} <= set(table[f"N={N},K={K},epi=store"])
