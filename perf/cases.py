"""What a user of the engine has it do, as cases that can be timed and compared: prompts, decode steps of one and of
many sequences, a known turn appended to growing caches, and sampling, all through the public entry points and at the
full model's size (28 layers, vocabulary 151936).

A case is a dict of plain values:

  prefill  {"kind", "tokens", "room"}            prefill(): a prompt of `tokens` ids into caches with `room` spare slots
  step     {"kind", "ctx"}                       Megakernel.step(): one sequence at position `ctx`
  decode   {"kind", "batch", "ctx", "ragged"}    bind_sequences() + launch(): one step of `batch` sequences of up to `ctx`
                                                 cached positions (all of them `ctx` long unless `ragged`)
  turn     {"kind", "batch", "ctx", "steps"}     bind_sequences(append=True) + launch() per position: `steps` known tokens a
                                                 sequence are appended to its cache (a user's turn in a running chat)
  sample   {"kind", "rows", "top_k", "temperature"}   sample(): one token for each of `rows` rows of logits
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "qwen3-megakernel_b200"))

from qwen3mk import Megakernel, prefill, sampling, weights  # noqa: E402
from qwen3mk.kernel import HEAD_DIM, HIDDEN, INTER, KV_HEADS, LAYERS, Q_HEADS, VOCAB, SeqTable  # noqa: E402

MAX_POSITIONS = 8192      # RoPE rows of an engine unless its caller asks for more


def listed():
    return [
        # choosing the next token: one chat with the usual top-k, and a full batch over the whole vocabulary
        {"name": "sample_1_top50", "kind": "sample", "rows": 1, "top_k": 50, "temperature": 0.8},
        {"name": "sample_64_all", "kind": "sample", "rows": 64, "top_k": 0, "temperature": 0.8},
        # one interactive stream: the position the headline figure is quoted on, an ordinary chat, a long document
        {"name": "step_128", "kind": "step", "ctx": 128},
        {"name": "step_1000", "kind": "step", "ctx": 1000},
        {"name": "step_5000", "kind": "step", "ctx": 5000},
        # three chats whose users have just answered: eight known tokens each, one position at a time
        {"name": "turn_3_ragged", "kind": "turn", "batch": 3, "ctx": 900, "steps": 8},
        # serving batches: small, ragged in the middle, the largest configured one
        {"name": "decode_8_1024", "kind": "decode", "batch": 8, "ctx": 1024, "ragged": False},
        {"name": "decode_27_ragged", "kind": "decode", "batch": 27, "ctx": 2048, "ragged": True},
        {"name": "decode_64_1024", "kind": "decode", "batch": 64, "ctx": 1024, "ragged": False},
        # prompts: the shortest the prefix rule takes, an odd one with room to decode in, a long one
        {"name": "prefill_128", "kind": "prefill", "tokens": 128, "room": 0},
        {"name": "prefill_777", "kind": "prefill", "tokens": 777, "room": 256},
        {"name": "prefill_2048", "kind": "prefill", "tokens": 2048, "room": 0},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sample", "step", "turn", "decode", "decode", "prefill", "prefill"])
    if kind == "sample":
        return {"kind": kind, "rows": _log_int(rng, 1, 64), "top_k": rng.choice([0, 20, 50, 200]),
                "temperature": round(rng.uniform(0.5, 0.9), 3)}
    if kind == "step":
        return {"kind": kind, "ctx": _log_int(rng, 16, 8000)}
    if kind == "turn":
        return {"kind": kind, "batch": rng.randint(1, 3), "ctx": _log_int(rng, 16, 900), "steps": rng.randint(2, 8)}
    if kind == "decode":
        batch = _log_int(rng, 2, 64)
        return {"kind": kind, "batch": batch, "ctx": _log_int(rng, 64, min(4096, 65536 // batch)), "ragged": rng.random() < 0.6}
    return {"kind": kind, "tokens": _log_int(rng, 16, 2048), "room": rng.choice([0, 1, 64, 300])}


def _lengths(case):
    """Cached positions of every sequence: `ctx`, or spread from a quarter of it up to all of it."""
    batch, ctx = case["batch"], case["ctx"]
    if not case.get("ragged", True) or batch == 1:
        return [ctx] * batch
    return [max(1, ctx - (3 * ctx * b) // (4 * (batch - 1))) for b in range(batch)]


def _model(seed):
    """All the engine's weights as seeded random tensors, without the caches that come with them."""
    inputs = weights.synthetic(seed, "cuda", context=1)
    return {k: inputs[k] for k in weights.WEIGHT_NAMES}


def _cache(gen, positions, capacity=None):
    """A K and a V cache [layers, capacity, 8, 128].  K rows leave a head norm and V rows a projection of normalised
    activations, so their elements are of size one."""
    shape = (LAYERS, capacity or positions, KV_HEADS, HEAD_DIM)
    pair = [torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(generator=gen) for _ in range(2)]
    for t in pair:
        t[:, positions:].zero_()
    return pair


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(1_000_003 + seed)
    kind = case["kind"]
    ids = lambda *shape: torch.randint(VOCAB, shape, generator=gen, device="cuda", dtype=torch.int64)  # noqa: E731
    if kind == "sample":
        # the logits of a trained model are far from flat: a few words carry most of the weight (about 2 nats here)
        logits = 5.0 * torch.randn((case["rows"], VOCAB), generator=gen, device="cuda")
        return {"case": case, "logits": logits, "u": torch.rand(case["rows"], generator=gen, device="cuda"),
                "out": torch.empty(case["rows"], dtype=torch.int64, device="cuda")}
    w = _model(seed)
    if kind == "prefill":
        n = case["tokens"]
        mk = Megakernel(max_tokens=n, max_positions=MAX_POSITIONS)
        first = torch.zeros(1, dtype=torch.int64, device="cuda")
        prefill.prefill(w, first, engine=mk)      # loading: the engine holds its weights before the first prompt
        return {"case": case, "mk": mk, "w": w, "ids": ids(n)}
    if kind == "step":
        mk = Megakernel(max_positions=MAX_POSITIONS)
        kc, vc = _cache(gen, case["ctx"])
        inputs = dict(w, token=ids(), kcache=kc, vcache=vc)
        mk.bind(inputs)                           # loading, as above
        return {"case": case, "mk": mk, "inputs": inputs}
    lens = _lengths(case)
    batch, room = case["batch"], case.get("steps", 0)
    caches = [_cache(gen, n, n + room) for n in lens]
    kcs, vcs = [c[0] for c in caches], [c[1] for c in caches]
    mk = Megakernel(max_batch=batch, max_positions=MAX_POSITIONS)
    tokens = ids(batch)
    s = {"case": case, "mk": mk, "w": w, "kcs": kcs, "vcs": vcs, "lens": lens, "tokens": tokens}
    seqs = SeqTable(kcs, vcs, lens)
    out = mk.bind_sequences(w, tokens, seqs)
    if kind == "turn":
        s["turn"] = ids(room, batch)
    else:
        s["out"] = out
    return s


def run(state):
    kind = state["case"]["kind"]
    if kind == "sample":
        c = state["case"]
        return sampling.sample(state["logits"], c["temperature"], c["top_k"], u=state["u"], out=state["out"])
    mk = state["mk"]
    if kind == "prefill":
        c = state["case"]
        return prefill.prefill(state["w"], state["ids"], capacity=c["tokens"] + c["room"], engine=mk)
    if kind == "step":
        return mk.step(state["inputs"])
    if kind == "decode":
        mk.launch()
        return state["out"]
    steps, lens = state["case"]["steps"], state["lens"]
    out = mk.bind_sequences(state["w"], state["tokens"], SeqTable(state["kcs"], state["vcs"], lens), append=True)
    for i in range(steps):
        state["tokens"].copy_(state["turn"][i])
        mk.launch()
    rows = [[c[:, n:n + steps] for c, n in zip(side, lens)] for side in (state["kcs"], state["vcs"])]
    return {"logits": out["logits"], "next_token": out["next_token"], "k_rows": rows[0], "v_rows": rows[1]}


_PER_LAYER = 2 * Q_HEADS * HEAD_DIM * HIDDEN + 2 * KV_HEADS * HEAD_DIM * HIDDEN + 3 * INTER * HIDDEN   # matrix elements
_GAINS = LAYERS * (2 * HIDDEN + 2 * HEAD_DIM) + HIDDEN
_KV_ROW = LAYERS * 2 * KV_HEADS * HEAD_DIM * 2        # bytes of one position's K and V rows


def _decode_work(lens):
    """One decode step: every weight, every cached row and one embedding row a sequence read once; logits and new rows written."""
    batch = len(lens)
    weight_bytes = 2 * (LAYERS * _PER_LAYER + VOCAB * HIDDEN + _GAINS)
    per_seq = 2 * HIDDEN + 4 * VOCAB + _KV_ROW + 16
    flops = 2 * batch * (LAYERS * _PER_LAYER + VOCAB * HIDDEN) + sum(4 * LAYERS * Q_HEADS * HEAD_DIM * (n + 1) for n in lens)
    return weight_bytes + sum(n * _KV_ROW for n in lens) + batch * per_seq, flops


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": case["rows"] * (4 * VOCAB + 12), "flops": 4 * case["rows"] * VOCAB}
    if kind == "prefill":
        n = case["tokens"]
        read = 2 * (LAYERS * _PER_LAYER + VOCAB * HIDDEN + _GAINS) + n * (8 + 2 * HIDDEN)
        written = (n + case["room"]) * _KV_ROW + 4 * VOCAB
        flops = 2 * n * LAYERS * _PER_LAYER + 2 * VOCAB * HIDDEN + 2 * LAYERS * Q_HEADS * HEAD_DIM * n * (n + 1)
        return {"bytes": read + written, "flops": flops}
    if kind == "step":
        b, f = _decode_work([case["ctx"]])
        return {"bytes": b, "flops": f}
    lens = _lengths(case)
    parts = [_decode_work([n + i for n in lens]) for i in range(case.get("steps", 1))]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        # at this temperature a row's rounding errors straddle the target once in about 1e5 rows
        return "exact"
    if kind == "prefill":
        # activations enter the products as bf16: the same inputs twice differ by 5e-3 (sums in another order, then other
        # roundings), an fp32 forward by 9e-3, single values by up to 0.05
        return {"rel": 2e-2, "max": 0.2, "differ": 0.01}
    # logits of two kernels differ by 2e-5, the bf16 K/V rows by 2e-4 (one unit in the last place, rarely), single values by 0.008
    return {"rel": 8e-4, "max": 0.032, "differ": 0.01}
