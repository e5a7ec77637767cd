"""The work that this framework is used for, as cases whose time can be measured.

Every case is one call of a public entry point of ``sageattention_b200`` on bf16 tensors: the dense operator
(``sageattn``), the K-packing operator (``sageattn4_blackwell``), packed variable-length batches
(``sageattn_varlen``) and the entry point for tensors in host memory (``sageattn_from_host``).  Values have the
distributions of the benchmark configurations: N(0,1), a per-channel offset on all keys (the outliers that K smoothing
removes) and, where video models have them, a few strong V channels.
"""
import math
import random

import torch

import sageattention_b200 as sa


def _case(name, op, B, Hq, Hkv, Nq, Nk, D, causal=False, layout="HND", lse=False, v_outliers=False):
    return {"name": name, "op": op, "B": B, "Hq": Hq, "Hkv": Hkv, "Nq": Nq, "Nk": Nk, "D": D, "causal": causal,
            "layout": layout, "lse": lse, "v_outliers": v_outliers}


def listed():
    return [
        # the first forward of a short prompt in a language model: launches and host work, hardly any arithmetic
        _case("short_prompt", "dense", 1, 32, 8, 128, 128, 128, causal=True),
        # the smallest of the benchmark configurations
        _case("small", "dense", 1, 8, 8, 1024, 1024, 128),
        # one decoding step of a batch against its cached keys, as a patched scaled_dot_product_attention sees it
        _case("decode", "dense", 8, 32, 8, 1, 4096, 128),
        # cross attention of an image model to a text: few keys, ragged lengths, a head dim between the native two, NHD
        _case("cross", "dense", 2, 16, 16, 4100, 333, 96, layout="NHD"),
        # the head dim 64 of the kernel sweep, at an image model's length
        _case("image_d64", "dense", 4, 32, 32, 4096, 4096, 64),
        # a serving batch of prompts of different lengths, packed (B sequences, Nk = the longest of them)
        _case("varlen", "varlen", 16, 32, 8, 3000, 3000, 128, causal=True),
        # the K-packing operator on a training-length context
        _case("k_packing", "packed", 4, 32, 32, 2048, 2048, 128, causal=True),
        # one step of ring attention over eight sequence shards of a long video: NHD shard, log-sum-exp for the merge
        _case("ring_step", "dense", 1, 40, 40, 9450, 9450, 128, layout="NHD", lse=True),
        # causal prefill with grouped query heads, from device and from pinned host memory
        _case("prefill", "dense", 4, 32, 8, 8192, 8192, 128, causal=True),
        _case("prefill_host", "host", 4, 32, 8, 8192, 8192, 128, causal=True),
        # self attention of a video diffusion transformer, the headline configuration
        _case("dit", "dense", 1, 40, 40, 32760, 32760, 128, v_outliers=True),
        # the long-sequence configuration on one GPU
        _case("long", "dense", 1, 40, 40, 75600, 75600, 128),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    op = rng.choice(["dense", "dense", "dense", "dense", "decode", "varlen", "packed", "host"])
    D = rng.choice([128, 128, 64]) if op != "dense" else rng.choice([128, 128, 128, 64, 64, 96, 72])
    if op == "decode":
        Hkv, Nq = rng.choice([4, 8, 32]), rng.choice([1, 1, 1, 2, 5, 16])
        return _drawn("dense", _log_uniform(rng, 1, 32), rng.choice([32, 32, 64]) if Hkv < 32 else 32, Hkv, Nq,
                      _log_uniform(rng, 256, 16384), D, Nq > 1, "HND", False)
    Hkv = rng.choice([4, 8, 16, 32])
    Hq = Hkv * rng.choice([1, 1, 2, 4]) if Hkv < 32 else Hkv
    causal = rng.random() < 0.5
    if op == "varlen":
        N = _log_uniform(rng, 64, 8192)
        B = _log_uniform(rng, 2, max(3, min(64, 65536 // N)))
        return _drawn(op, B, Hq, Hkv, N, N, D, causal, "NHD", False)
    if op == "packed":
        N = _log_uniform(rng, 100, 8192)
        return _drawn(op, _log_uniform(rng, 1, max(2, min(8, 16384 // N))), Hq, Hkv, N, N, D, causal, rng.choice(["HND", "NHD"]), False)
    if op == "host":
        N = _log_uniform(rng, 256, 16384)
        return _drawn(op, _log_uniform(rng, 1, max(2, min(8, 16384 // N))), Hq, Hkv, N, N, D, causal, "HND", False)
    Nq = _log_uniform(rng, 64, 40000)
    # mostly self attention; else cross attention to fewer keys, or a chunk of queries behind cached keys
    Nk = Nq if rng.random() < 0.6 else _log_uniform(rng, 77, min(16384, 2 ** 29 // Nq))
    if Nk < Nq:
        causal = False
    B = _log_uniform(rng, 1, max(2, min(8, 65536 // max(Nq, Nk))))
    return _drawn(op, B, Hq, Hkv, Nq, Nk, D, causal, rng.choice(["HND", "NHD"]), rng.random() < 0.25)


def _drawn(*args):
    c = _case("", *args)
    del c["name"]
    return c


def _lengths(case):
    """Sequence lengths of a packed batch: the longest one first, the others spread over a factor of sixteen."""
    rng = random.Random(case["B"] * 1000003 + case["Nk"])
    n = case["Nk"]
    return [n] + [_log_uniform(rng, max(1, n // 16), n) for _ in range(case["B"] - 1)]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op, B, Hq, Hkv, D = case["op"], case["B"], case["Hq"], case["Hkv"], case["D"]
    nhd = case["layout"] == "NHD"

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)

    if op == "varlen":
        lens = _lengths(case)
        q, k, v = normal(sum(lens), Hq, D), normal(sum(lens), Hkv, D), normal(sum(lens), Hkv, D)
        k += 2.0 * normal(1, Hkv, D)
    else:
        def of(heads, n):
            return normal(B, n, heads, D) if nhd else normal(B, heads, n, D)
        q, k, v = of(Hq, case["Nq"]), of(Hkv, case["Nk"]), of(Hkv, case["Nk"])
        k += 2.0 * of(Hkv, 1)
    if case["v_outliers"]:
        v[..., torch.randperm(D, generator=g, device="cuda")[:max(1, D // 20)]] *= 8
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    state = {"case": case, "q": q, "k": k, "v": v}
    if op == "varlen":
        starts = [0]
        for n in lens:
            starts.append(starts[-1] + n)
        state["cu"] = torch.tensor(starts, dtype=torch.int32, device="cuda")
    elif op == "host":
        for name in "qkv":
            t = state[name]
            state[name] = torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)
        state["out"] = torch.empty(state["q"].shape, dtype=torch.bfloat16, pin_memory=True)
    return state


def run(state):
    case, q, k, v = state["case"], state["q"], state["k"], state["v"]
    if case["op"] == "varlen":
        return sa.sageattn_varlen(q, k, v, state["cu"], state["cu"], case["Nq"], case["Nk"], is_causal=case["causal"])
    if case["op"] == "packed":
        return sa.sageattn4_blackwell(q, k, v, tensor_layout=case["layout"], is_causal=case["causal"])
    if case["op"] == "host":
        return sa.sageattn_from_host(q, k, v, out=state["out"], is_causal=case["causal"])
    return sa.sageattn(q, k, v, tensor_layout=case["layout"], is_causal=case["causal"], return_lse=case["lse"])


def _pairs(nq, nk, causal):
    """Query-key pairs that attention visits; the causal diagonal is aligned to the last query and key."""
    if not causal:
        return nq * nk
    first = nk - nq + 1                       # keys that the first query sees
    rows = nq if first >= 1 else nk           # queries that see any key
    return rows * (max(first, 1) + nk) // 2


def work(case):
    B, Hq, Hkv, Nq, Nk, D = (case[n] for n in ("B", "Hq", "Hkv", "Nq", "Nk", "D"))
    seqs = [(n, n) for n in _lengths(case)] if case["op"] == "varlen" else [(Nq, Nk)] * B
    rows_q, rows_k = sum(a for a, _ in seqs), sum(b for _, b in seqs)
    return {"bytes": 2.0 * D * (2 * Hq * rows_q + 2 * Hkv * rows_k) + (4.0 * Hq * rows_q if case["lse"] else 0.0),
            "flops": 4.0 * Hq * D * sum(_pairs(a, b, case["causal"]) for a, b in seqs)}


def tolerance(case):
    # bf16 outputs of 4-bit operands: a last-bit difference in a channel mean moves some values across a rounding
    # boundary of the 4-bit grid
    return {"rel": 0.02, "max": 0.5}
