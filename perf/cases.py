"""What this framework is used for, as a list of measurable passes through its public entry points.

A pass is what one call (or one short run of calls) of a user's program does:

  decode   tokens of one sequence, one `RWKV.forward([id], state)` each, from the state that a prompt left
  batch    `RWKV.forward_batch` steps of B sequences at once
  prefill  a prompt through `RWKV.forward(ids, None)`, whole or in chunks that hand the state on
  score    a prompt with `full_output=True`: the logits of every position (perplexity, choice ranking)
  sample   the draws of one generation: a fresh `Sampler`, then one token per row of logits, as
           `PIPELINE.generate_tokens` does between its forward calls
  matmul   one call of `torch.ops.rwkv.mm8_one` / `mm8_seq` on a packed matrix

The models are the random-init shapes of `chatrwkv_b200.synth` (and the RWKV-5.2 width of the tests); a program loads
its model once, so the model of a shape is kept for the life of the process and only prompts, states, ids, logits and
operands are made anew from the seed.  Decoding is fed with given ids instead of its own arg-max: the work is the same
and the outputs stay comparable when two logits are nearly equal.
"""
import functools
import math

import torch

from chatrwkv_b200 import ops, synth
from chatrwkv_b200.model import RWKV
from chatrwkv_b200.pipeline import PIPELINE_ARGS, Sampler

# name: (version, n_layer, n_embd, n_ffn, vocab)
SHAPES = {
    "v4-169m": (4,) + synth.SHAPES["v4-169m"],
    "v4-7b": (4,) + synth.SHAPES["v4-7b"],
    "v5-7b": (5.2, 32, 4096, 14336, 65536),
    "v6-7b": (6,) + synth.SHAPES["v6-7b"],
}
MATRICES = ((4096, 4096), (4096, 16384), (16384, 4096), (5120, 20480))      # the operator sweep's shapes
HEAD = 64
PROMPT = 48              # tokens in the state before a decode or batch step


def listed():
    return [
        # one user, one token at a time: the smallest model (launches and host work show) ...
        {"name": "decode-v4-169m", "kind": "decode", "shape": "v4-169m", "tokens": 16},
        # ... the headline configuration of this repository ...
        {"name": "decode-v4-7b", "kind": "decode", "shape": "v4-7b", "tokens": 8},
        # ... and the family with data-dependent decay
        {"name": "decode-v6-7b", "kind": "decode", "shape": "v6-7b", "tokens": 8},
        # a served model: a few users at once, and the 64 sequences of the multi-sequence configuration
        {"name": "batch-v4-7b-16", "kind": "batch", "shape": "v4-7b", "rows": 16, "steps": 4},
        {"name": "batch-v6-7b-64", "kind": "batch", "shape": "v6-7b", "rows": 64, "steps": 2},
        # a short chat message on the smallest model
        {"name": "prefill-v4-169m-64", "kind": "prefill", "shape": "v4-169m", "tokens": 64, "chunk": 0},
        # a prompt in the generation loop's default chunks of 256, the last one ragged
        {"name": "prefill-v5-7b-600-chunks", "kind": "prefill", "shape": "v5-7b", "tokens": 600, "chunk": 256},
        # the headline configuration's prompt, and the long prompt of the multi-sequence configuration
        {"name": "prefill-v4-7b-1024", "kind": "prefill", "shape": "v4-7b", "tokens": 1024, "chunk": 0},
        {"name": "prefill-v6-7b-2048", "kind": "prefill", "shape": "v6-7b", "tokens": 2048, "chunk": 0},
        # scoring a document of an odd length: logits of every position
        {"name": "score-v4-7b-333", "kind": "score", "shape": "v4-7b", "tokens": 333},
        # the sampler's share of a generation
        {"name": "sample-65536", "kind": "sample", "vocab": 65536, "draws": 32, "top_p": 0.85, "top_k": 0, "temperature": 1.0},
        # the operator by itself at one point of the sweep
        {"name": "matmul-16-4096-16384", "kind": "matmul", "rows": 16, "n": 4096, "m": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "batch", "prefill", "prefill", "score", "sample", "matmul", "matmul"))
    shape = rng.choice(sorted(SHAPES))
    if kind == "decode":
        return {"kind": kind, "shape": shape, "tokens": rng.randint(2, 16)}
    if kind == "batch":
        return {"kind": kind, "shape": shape, "rows": _log_int(rng, 2, 64), "steps": rng.randint(1, 4)}
    if kind == "prefill":
        # a v6 prompt of 2048 tokens is the largest case there is
        return {"kind": kind, "shape": shape, "tokens": _log_int(rng, 2, 1900), "chunk": rng.choice((0, 0, 256))}
    if kind == "score":
        # RWKV-4: the group norm of the other families divides by nearly nothing at the first positions, so that their
        # logits there say more about the last bit than about the path (random weights)
        return {"kind": kind, "shape": rng.choice(("v4-169m", "v4-7b")), "tokens": _log_int(rng, 8, 512)}
    if kind == "sample":
        return {"kind": kind, "vocab": rng.choice((50277, 65536, rng.randint(20000, 65536))), "draws": rng.randint(8, 32),
                "top_p": rng.choice((0.3, 0.5, 0.85, 1.0)), "top_k": rng.choice((0, 0, 40)), "temperature": rng.choice((0.7, 1.0, 1.2))}
    n, m = rng.choice(MATRICES)
    return {"kind": kind, "rows": _log_int(rng, 1, 1024), "n": n, "m": m}


@functools.lru_cache(maxsize=None)
def _model(shape):
    version, n_layer, n_embd, n_ffn, vocab = SHAPES[shape]
    ck = synth.make_checkpoint(version, n_layer, n_embd, n_ffn, vocab, seed=1, head_size=HEAD, device="cuda", dtype=torch.float16)
    return RWKV(ck, "cuda fp16i8", verbose=False)


def _own(state):
    """A state list in tensors of its own (the model's persistent buffers are written by its next call)."""
    return [t.clone() for t in state]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("matmul", "sample"):
        g = torch.Generator(device="cuda").manual_seed(seed)
        if kind == "matmul":
            rows, n, m = case["rows"], case["n"], case["m"]
            packed = ops.quantize_weight(torch.randn(n, m, generator=g, device="cuda") * 0.02)
            x = torch.randn(rows, n, generator=g, device="cuda").half()
            return {"case": case, "x": x, "packed": packed}
        v = case["vocab"]
        # a trained model's logits: a bulk, and a handful of likely ids per row
        logits = torch.randn(case["draws"], v, generator=g, device="cuda") * 2.0
        likely = torch.randint(0, v, (case["draws"], 32), generator=g, device="cuda")
        logits.scatter_add_(1, likely, torch.rand(case["draws"], 32, generator=g, device="cuda") * 12.0)
        args = PIPELINE_ARGS(temperature=case["temperature"], top_p=case["top_p"], top_k=case["top_k"], token_ban=[0])
        return {"case": case, "logits": logits, "args": args, "seed": seed}
    model = _model(case["shape"])
    vocab = SHAPES[case["shape"]][4]
    if kind in ("prefill", "score"):
        return {"case": case, "model": model, "ids": synth.make_tokens(case["tokens"], vocab, seed)}
    if kind == "decode":
        _, state = model.forward(synth.make_tokens(PROMPT, vocab, seed), None)
        return {"case": case, "model": model, "state": _own(state), "ids": synth.make_tokens(case["tokens"], vocab, seed + 1)}
    rows, steps = case["rows"], case["steps"]
    ids = torch.tensor(synth.make_tokens(rows * (steps + 2), vocab, seed + 1), device="cuda").view(steps + 2, rows)
    # two prompts of their own for the first rows' states, then two batched tokens that set all rows apart
    starts = [model.forward(synth.make_tokens(PROMPT, vocab, seed + 2 + k), None)[1] for k in range(2)]
    state = model.stack_states([starts[b % 2] for b in range(rows)])
    for k in range(2):
        _, state = model.forward_batch(ids[k], state)
    return {"case": case, "model": model, "state": _own(state), "ids": ids[2:]}


def _packed_state(state, per_layer):
    """The state list as one tensor per kind of entry (how a program that keeps many sessions stores it)."""
    return [torch.stack(state[j::per_layer]) for j in range(per_layer)]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "matmul":
        x, packed = state["x"], state["packed"]
        rows, n, m = case["rows"], case["n"], case["m"]
        if rows == 1:
            y = torch.zeros(m, dtype=torch.float32, device=x.device)
            torch.ops.rwkv.mm8_one(n, m, x[0], *packed, y)
        else:
            y = torch.empty((rows, m), dtype=x.dtype, device=x.device)
            torch.ops.rwkv.mm8_seq(rows, n, m, x, *packed, y)
        return y
    if kind == "sample":
        logits = state["logits"]
        sampler = Sampler(logits.shape[1], logits.device, state["args"], state["seed"])
        ids = torch.zeros(len(logits), dtype=torch.int64, device=logits.device)
        for i in range(len(logits)):
            ids[i:i + 1].copy_(sampler.sample(logits[i]))
        return ids, sampler.occurrence
    model, ids = state["model"], state["ids"]
    per_layer = 5 if model.version == 4 else 3
    if kind == "score":
        logits, st = model.forward(ids, None, full_output=True)
        return logits, _packed_state(st, per_layer)
    if kind == "prefill":
        st, chunk = None, case["chunk"] or len(ids)
        for at in range(0, len(ids), chunk):
            logits, st = model.forward(ids[at:at + chunk], st)
        return logits, _packed_state(st, per_layer)
    st, out = state["state"], []
    for i in range(len(ids)):
        if kind == "decode":
            logits, st = model.forward([ids[i]], st)
        else:
            logits, st = model.forward_batch(ids[i], st)
        out.append(logits)
    return out, _packed_state(st, per_layer)


def _sizes(shape):
    """(bytes of codes and scales without the head's, multiplications of them per token, the same two of the head, bytes
    of one sequence's state)."""
    version, layers, d, f, vocab = SHAPES[shape]
    square = 5 if version == 4 else 6                     # d x d matrices: receptance, key, value, output (, gate), ffn.receptance
    packed = lambda n, m: n * m + 4 * (n + m)             # noqa: E731  codes, fp16 mx, rx, my, ry
    body = layers * (square * packed(d, d) + packed(d, f) + packed(f, d))
    mults = layers * (square * d * d + 2 * d * f)
    if version == 6:
        low = d * 10 * synth.V6_MAA_RANK + 2 * d * synth.V6_DECAY_RANK
        body, mults = body + layers * 2 * low, mults + layers * low
    state = layers * (4 * d + (12 * d if version == 4 else 4 * d * HEAD))
    return body, mults, packed(d, vocab), d * vocab, state


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        rows, n, m = case["rows"], case["n"], case["m"]
        return {"bytes": n * m + 4 * (n + m) + rows * (2 * n + (4 if rows == 1 else 2) * m), "flops": 2 * rows * n * m}
    if kind == "sample":
        v, draws = case["vocab"], case["draws"]
        return {"bytes": draws * 14 * v, "flops": draws * 8 * v}      # logits; occurrence and marks in and out per draw
    body, mults, head, head_mults, state = _sizes(case["shape"])
    vocab = SHAPES[case["shape"]][4]
    if kind in ("decode", "batch"):      # every step needs the step before it: the weights are read once a step
        rows, steps = (1, case["tokens"]) if kind == "decode" else (case["rows"], case["steps"])
        return {"bytes": steps * (body + head + rows * (2 * state + 4 * vocab)), "flops": 2 * steps * rows * (mults + head_mults)}
    tokens = case["tokens"]
    chunks = -(-tokens // case["chunk"]) if case.get("chunk") else 1
    rows = tokens if kind == "score" else chunks           # positions whose logits are computed
    return {"bytes": chunks * (body + head) + state + 4 * vocab * rows, "flops": 2 * (tokens * mults + rows * head_mults)}


# Four times what the path differs from itself when the fp32 arithmetic of another of its kernels takes the place of
# the default one: fp16 activations are rounded at every operation, and one flipped rounding spreads through the layers.
_TOLERANCE = {
    "v4-169m": {"rel": 4.5e-3, "max": 2.2e-2},      # seen: 1.1e-3, 5.3e-3
    "v4-7b": {"rel": 1.4e-2, "max": 7e-2},          # seen: 3.5e-3, 1.7e-2
    "v5-7b": {"rel": 2.3e-2, "max": 0.16},          # seen at v6-7b: 5.6e-3, 3.9e-2 (group norms of small heads)
    "v6-7b": {"rel": 2.3e-2, "max": 0.16},
}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    if kind == "matmul":
        return {"rel": 2e-4, "max": 4e-3}            # seen: 4e-5, 1e-3 (single roundings to fp16 that fall the other way)
    return _TOLERANCE[case["shape"]]
