"""The work that users of this package have it do, as measurable cases.

``listed()`` names representative calls of every path -- single decode FCs, a batch of independent FCs, a token
through a block stack, prefill, weight packing, the per-channel int8 FC and the embedding look-up -- and ``draw()``
gives further ones over the same ranges of sizes and block types.  Everything goes through the public entry points
(``llmops``, ``ops``, ``host``, ``stack``).  Weights are N(0, 0.02) and activations N(0, 1), as in ``bench.py``.
"""
from __future__ import annotations

import math

import torch

import llama_cl_b200 as pkg

GROUPS = (32, 128)
MOST_WEIGHTS = 4096 * 32000           # the largest weight tensor: lm_head of Llama-7B
MOST_MACS = 2048 * 4096 * 11008       # the largest contraction: a 2048-token prompt through an up projection


# ------------------------------------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # one attention projection for one token in the stock block type: the smallest call, all latency
        dict(name="fc_1row_q41_g32", kind="fc", rows=1, K=4096, N=4096, qtype="q4_1", group_k=32),
        # a program that keeps its activations in host memory, as the reference's users do: lm_head of one token
        dict(name="host_lm_head_1row", kind="host", rows=1, K=4096, N=32000, qtype="q4_1", group_k=128),
        # an nn.Linear replacement with bias whose sizes fit no tile, for a few sequences at once
        dict(name="linear_3rows_ragged", kind="linear", rows=3, K=3001, N=5003, qtype="q4_0", group_k=32),
        # the benchmark's decode sweep: four Llama-7B shapes at 1, 2, 4 and 8 rows, independent calls batched
        dict(name="batch_sweep", kind="batch", rows="8,4,2,1", hidden=4096, intermediate=11008, vocab=32000,
             qtype="q4_1", group_k=128),
        # one generated token through Llama-7B-wide layers and lm_head, waited for because the next token needs it
        dict(name="token_4layers", kind="stack", rows=1, layers=4, hidden=4096, intermediate=11008, vocab=32000,
             qtype="q4_1", group_k=128),
        # a short prompt (or many sequences decoding together) through an up projection
        dict(name="prefill_37rows_q41_g32", kind="fc", rows=37, K=4096, N=11008, qtype="q4_1", group_k=32),
        # an ordinary prompt: the benchmark's prefill configuration
        dict(name="prefill_512rows_q40_g32", kind="fc", rows=512, K=4096, N=11008, qtype="q4_0", group_k=32),
        # a long prompt, the largest contraction, in the block type of the decode configurations
        dict(name="prefill_2048rows_q41_g128", kind="fc", rows=2048, K=4096, N=11008, qtype="q4_1", group_k=128),
        # loading a model: one down projection packed
        dict(name="pack_q41_g128", kind="pack", K=11008, N=4096, qtype="q4_1", group_k=128),
        # per-channel int8 weights (the older extension's FC): lm_head of one token ...
        dict(name="q8c_1row", kind="q8c", rows=1, K=4096, N=32000),
        # ... and a prompt
        dict(name="q8c_256rows", kind="q8c", rows=256, K=4096, N=11008),
        # the token table of a prompt of 2048 tokens
        dict(name="embedding_2048ids", kind="embedding", ids=2048, V=32000, E=4096),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _size(rng, lo: int, hi: int) -> int:
    """A dimension: half of them multiples of 128, as model widths are, the others anything."""
    v = _log(rng, lo, hi)
    return max(128, v // 128 * 128) if rng.random() < 0.5 else v


def _matrix(rng) -> dict:
    K = _size(rng, 512, 11008)
    return dict(K=K, N=_size(rng, 512, min(32000, MOST_WEIGHTS // K)))


def draw(rng) -> dict:
    kind = rng.choice(["fc", "fc", "prefill", "prefill", "host", "linear", "batch", "stack", "pack", "q8c", "embedding"])
    block = dict(qtype=rng.choice(["q4_0", "q4_1"]), group_k=rng.choice(GROUPS))
    if kind == "fc":
        return dict(kind="fc", rows=rng.randint(1, 8), **_matrix(rng), **block)
    if kind == "prefill":
        m = _matrix(rng)
        return dict(kind="fc", rows=_log(rng, 9, min(2048, MOST_MACS // (m["K"] * m["N"]))), **m, **block)
    if kind in ("host", "linear"):
        return dict(kind=kind, rows=rng.randint(1, 8), **_matrix(rng), **block)
    if kind == "batch":
        rows = sorted(rng.sample(range(1, 9), rng.randint(1, 4)), reverse=True)
        hidden = _log(rng, 1024, 4096) // 32 * 32
        return dict(kind="batch", rows=",".join(map(str, rows)), hidden=hidden,
                    intermediate=int(hidden * rng.uniform(2.0, 2.6875)) // 8 * 8, vocab=_log(rng, 2000, 32000), **block)
    if kind == "stack":
        hidden = _log(rng, 1024, 4096) // 32 * 32
        return dict(kind="stack", rows=rng.randint(1, 4), layers=rng.randint(1, 4), hidden=hidden,
                    intermediate=int(hidden * rng.uniform(2.0, 2.6875)) // 32 * 32, vocab=_log(rng, 2000, 32000), **block)
    if kind == "pack":
        return dict(kind="pack", **_matrix(rng), **block)
    if kind == "q8c":
        return dict(kind="q8c", rows=_log(rng, 1, 512), **_matrix(rng))
    return dict(kind="embedding", ids=_log(rng, 1, 4096), V=_log(rng, 2000, 32000), E=_size(rng, 512, 4096))


# ------------------------------------------------------------------------------------------------ inputs
class _Source:
    """Seeded weights and activations on the GPU."""

    def __init__(self, seed: int) -> None:
        self.dev = torch.device("cuda")
        self.gen = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape) -> torch.Tensor:
        return torch.randn(*shape, generator=self.gen, device=self.dev)

    def weight(self, N: int, K: int) -> torch.Tensor:
        return self.normal(N, K).mul_(0.02)

    def packed(self, N: int, K: int, case: dict) -> torch.Tensor:
        return pkg.llmops.offline_FC_quant_Q4A(self.weight(N, K), qtype=case["qtype"], group_k=case["group_k"])


def _batch_shapes(case: dict) -> list[tuple[int, int]]:
    H, I, V = case["hidden"], case["intermediate"], case["vocab"]
    return [(H, H), (H, I), (I, H), (H, V)]  # (K, N)


def prepare(case: dict, seed: int):
    src, ops, kind = _Source(seed), pkg.llmops, case["kind"]
    if kind == "fc":
        w = src.packed(case["N"], case["K"], case)
        return dict(kind=kind, w=w, N=case["N"], x=src.normal(1, case["rows"], case["K"]))
    if kind == "host":
        fc = pkg.host.HostFC(src.packed(case["N"], case["K"], case), case["N"])
        # the program's own activations, in ordinary host memory (HostFC takes K as packed: whole groups)
        x = torch.zeros(1, case["rows"], fc.K)
        x[:, :, : case["K"]] = src.normal(1, case["rows"], case["K"]).cpu()
        return dict(kind=kind, fc=fc, x=x)
    if kind == "linear":
        lin = torch.nn.Linear(case["K"], case["N"], device="meta")
        lin.weight = torch.nn.Parameter(src.weight(case["N"], case["K"]), requires_grad=False)
        lin.bias = torch.nn.Parameter(src.normal(case["N"]), requires_grad=False)
        op = pkg.ops.llmop_fc_q4a(lin, qtype=case["qtype"], group_k=case["group_k"])
        return dict(kind=kind, op=op, x=src.normal(1, case["rows"], case["K"]))
    if kind == "batch":
        launches = []
        for rows in map(int, case["rows"].split(",")):
            pairs, calls = [], []
            for K, N in _batch_shapes(case):
                xq = ops.QuantizedActivations(1, rows, K, case["group_k"], False, src.dev)
                pairs.append((src.normal(1, rows, K), xq))
                calls.append((xq, src.packed(N, K, case), N))
            launches.append((ops.QuantizeBatch(pairs), ops.FCBatch(calls, pdl=True)))
        return dict(kind=kind, launches=launches)
    if kind == "stack":
        H, I, V = case["hidden"], case["intermediate"], case["vocab"]
        sizes = dict(q=(H, H), k=(H, H), v=(H, H), o=(H, H), gate=(I, H), up=(I, H), down=(H, I))
        layers = [{k: src.packed(N, K, case) for k, (N, K) in sizes.items()} for _ in range(case["layers"])]
        norms = [dict(input=src.normal(H).mul_(0.1).add_(1), post=src.normal(H).mul_(0.1).add_(1))
                 for _ in range(case["layers"])]
        stack = pkg.stack.DecodeFCStack(layers, src.packed(V, H, case), hidden=H, intermediate=I, vocab=V,
                                        rows=case["rows"], norms=norms)
        return dict(kind=kind, stack=stack, x=src.normal(1, case["rows"], H))
    if kind == "pack":
        return dict(kind=kind, w=src.weight(case["N"], case["K"]), qtype=case["qtype"], group_k=case["group_k"])
    if kind == "q8c":
        w, scales = pkg.c_ext.FC_quant_Q8C(src.weight(case["N"], case["K"]))
        return dict(kind=kind, w=w, scales=scales, N=case["N"], x=src.normal(1, case["rows"], case["K"]))
    if kind == "embedding":
        op = pkg.ops.llmop_embedding_q8c(src.weight(case["V"], case["E"]))
        ids = torch.randint(0, case["V"], (1, case["ids"]), generator=src.gen, device=src.dev)
        return dict(kind=kind, op=op, ids=ids)
    raise ValueError(f"unknown kind {kind!r}")


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "fc":
        return pkg.llmops.fc_Q4A(state["x"], state["w"], state["N"])
    if kind == "host":
        return state["fc"](state["x"])
    if kind == "linear":
        return state["op"](state["x"])
    if kind == "batch":
        for quantize, fcs in state["launches"]:
            quantize.run()
            fcs.run()
        return [fcs.outs for _, fcs in state["launches"]]
    if kind == "stack":
        return state["stack"].forward(state["x"], sync=True)  # the next token is sampled from the logits
    if kind == "pack":
        return pkg.llmops.offline_FC_quant_Q4A(state["w"], qtype=state["qtype"], group_k=state["group_k"])
    if kind == "q8c":
        return pkg.c_ext.FC_evaluate_Q8C(state["x"], state["w"], state["scales"], state["N"])
    return state["op"](state["ids"])


# ------------------------------------------------------------------------------------------------ what a pass costs
def _packed_bytes(K: int, N: int, case: dict) -> int:
    G = case["group_k"]
    return -(-N // 32) * -(-K // G) * (16 * G + (128 if case["qtype"] == "q4_1" else 64))


def _fc_work(K: int, N: int, rows: int, case: dict) -> tuple[int, int]:
    return _packed_bytes(K, N, case) + 4 * rows * (K + N), 2 * rows * N * K


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("fc", "host", "linear"):
        nbytes, flops = _fc_work(case["K"], case["N"], case["rows"], case)
        nbytes += 4 * case["N"] if kind == "linear" else 0
    elif kind == "batch":
        each = [_fc_work(K, N, int(r), case) for r in case["rows"].split(",") for K, N in _batch_shapes(case)]
        nbytes, flops = sum(b for b, _ in each), sum(f for _, f in each)
    elif kind == "stack":
        H, I, V, L, R = (case[k] for k in ("hidden", "intermediate", "vocab", "layers", "rows"))
        mats = [(H, H)] * (4 * L) + [(H, I)] * (2 * L) + [(I, H)] * L + [(H, V)]
        nbytes = sum(_packed_bytes(K, N, case) for K, N in mats) + 4 * R * (H + V) + 4 * H * (2 * L + 1)
        flops = 2 * R * sum(K * N for K, N in mats)
    elif kind == "pack":
        nbytes, flops = 4 * case["N"] * case["K"] + _packed_bytes(case["K"], case["N"], case), 0
    elif kind == "q8c":
        N, K, R = case["N"], case["K"], case["rows"]
        nbytes, flops = -(-N // 32) * -(-K // 32) * 1024 + 4 * N + 4 * R * (K + N), 2 * R * N * K
    else:
        nbytes, flops = case["ids"] * (8 + 4 + 5 * case["E"]), 0
    return dict(bytes=nbytes, flops=flops)


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("pack", "embedding"):
        return "exact"  # bytes, and one product per value
    if kind == "stack":
        # every FC quantizes its input to 8 bits again: a sum that differs in its last place can move a code by one
        # step (1/127 of its group's largest value), and the layers behind it see that
        return dict(rel=5e-3)
    return dict(rel=1e-5)  # exact integer dots, fp32 sums over the groups
