"""The work that users of this package have it do, as cases that can be timed: a case says what, ``prepare`` makes the
inputs and whatever a program keeps between calls, ``run`` is one pass through the public entry points of
``kiln_b200.api``.

Kinds of work, by the ``kind`` of a case:

  verify    the speculative round: k drafted tokens per sequence and one more row, greedy rows, acceptance
            (``verify_step``); with k = 0 a synchronous decode step
  decode    two pipelined decode steps, the second fed from the first on the device (``decode_launch`` / ``decode_collect``)
  forward   one forward pass over a mixed batch with its logits (``forward_step``): a prompt chunk, rows of running
            sequences, or both
  draft     a draft model's chain of k one-row forwards (``draft_chain``)
  linear    one quantised linear (``QuantizedWeight.matmul``)
  attention paged attention on its own (``paged_attention``)

Weights are random: layers N(0, 0.01), quantised by ``kiln_b200.synth``; a layer adds a tenth or so to the residual
stream, as a trained one does (with larger weights a random model multiplies every rounding from layer to layer). The
head is a permutation of the embedding (or tied to it), so that every next token has a clear winner, as a trained
model's mostly have, and a draft can be right with a chosen probability. A history in the cache is one
prompt's, run through the model; the other sequences hold copies of its blocks, in blocks of their own.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from kiln_b200 import api
from kiln_b200.synth import PRESETS, quantize_affine, synth_checkpoint, truncated

BLOCK = 16        # tokens in a block of the paged cache
CHUNK = 2048      # prompt tokens of one forward, and the step size that the models are loaded for
ACCEPT = 0.7      # share of drafted tokens that are the target's own choice


def listed():
    return [
        # The smallest whole-model call: a draft model (4 layers of the 1B architecture, weight-streaming lane on)
        # proposing for one sequence.
        dict(name="draft_1b4l_k4", kind="draft", model="llama-3.2-1b", layers=4, batch=1, k=4, lo=190, hi=190, shared=0, piece=0, start=0),
        # One interactive user on a small model: five rows, launch latency counts.
        dict(name="verify_1b_k4_bs1", kind="verify", model="llama-3.2-1b", layers=16, batch=1, k=4, lo=190, hi=190, shared=0, piece=0, start=0),
        # One user on an 8B model, plain decode: every weight is read for one row.
        dict(name="forward_8b_bs1", kind="forward", model="llama-3.1-8b", layers=32, batch=1, k=0, lo=1001, hi=1001, shared=0, piece=0, start=0),
        # A full server without speculation, pipelined.
        dict(name="decode_8b_bs32", kind="decode", model="llama-3.1-8b", layers=32, batch=32, k=0, lo=512, hi=2048, shared=0, piece=0, start=0),
        # The headline: a full server with speculation.
        dict(name="verify_8b_k5_bs32", kind="verify", model="llama-3.1-8b", layers=32, batch=32, k=5, lo=512, hi=2048, shared=0, piece=0, start=0),
        # The second half of a 4096-token prompt.
        dict(name="prefill_8b_2048", kind="forward", model="llama-3.1-8b", layers=32, batch=0, k=0, lo=0, hi=0, shared=0, piece=2048, start=2048),
        # Continuous batching: an odd piece of a new prompt rides along with the rows of running sequences.
        dict(name="mixed_8b_333_bs11", kind="forward", model="llama-3.1-8b", layers=32, batch=11, k=2, lo=100, hi=1500, shared=0, piece=333, start=0),
        # 8-bit weights, groups of 32; requests that share a system prompt, 320 rows.
        dict(name="verify_7b_w8_k4_bs64", kind="verify", model="qwen2.5-7b", layers=28, batch=64, k=4, lo=1280, hi=1280, shared=1024, piece=0, start=0),
        # Groups of 128, head size 256, soft caps, sliding window; long contexts.
        dict(name="forward_9b_k3_bs16", kind="forward", model="gemma-2-9b", layers=42, batch=16, k=3, lo=6144, hi=6144, shared=0, piece=0, start=0),
        # The widest layers (8 of them), long ragged contexts, 320 rows.
        dict(name="forward_70b8l_k4_bs64", kind="forward", model="llama-3-70b-8l", layers=8, batch=64, k=4, lo=1024, hi=4096, shared=0, piece=0, start=0),
        # One linear of a caller's own graph, no size a multiple of a tile.
        dict(name="linear_w4_m37", kind="linear", model="", bits=4, group=64, rows=37, n_out=11000, n_in=4096),
        # Attention of a caller's own graph, ragged.
        dict(name="attention_bs8_q6", kind="attention", model="", heads=32, kv_heads=8, head_dim=128, batch=8, k=5, lo=300, hi=3000),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm, odd ones as likely as even ones."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


_DRAWN = {  # layers, and the cached tokens over all sequences that keep a drawn case below the largest listed one
    "llama-3.2-1b": (16, 60000), "llama-3.1-8b": (32, 45000), "qwen2.5-7b": (28, 60000), "gemma-2-9b": (42, 50000), "llama-3-70b-8l": (8, 120000)}


def draw(rng):
    kind = rng.choice(["verify", "verify", "verify", "decode", "forward", "forward", "forward", "draft", "linear", "attention"])
    if kind == "linear":
        bits, group = rng.choice([(4, 64), (4, 128), (4, 32), (8, 32), (8, 64)])
        n_in = 128 * _spread(rng, 8, 112)
        n_out = _spread(rng, 500, 30000)
        rows = _spread(rng, 1, 512)
        return dict(kind=kind, model="", bits=bits, group=group, rows=rows, n_out=n_out, n_in=n_in)
    if kind == "attention":
        head_dim, heads, kv_heads = rng.choice([(128, 32, 8), (64, 32, 8), (128, 28, 4), (256, 16, 8), (128, 64, 8)])
        batch = _spread(rng, 1, 48)
        hi = _spread(rng, 40, min(8000, 100000 // batch))
        return dict(kind=kind, model="", heads=heads, kv_heads=kv_heads, head_dim=head_dim, batch=batch, k=rng.randint(0, 6), lo=max(1, hi // 3), hi=hi)
    name = rng.choice(["llama-3.2-1b", "llama-3.1-8b"] if kind in ("draft", "decode") else list(_DRAWN))
    layers, tokens = _DRAWN[name]
    if kind == "draft":
        hi = _spread(rng, 20, 4000)
        return dict(kind=kind, model=name, layers=4, batch=1, k=rng.randint(1, 7), lo=hi, hi=hi, shared=0, piece=0, start=0)
    if kind == "forward" and rng.random() < 0.4:   # a prompt chunk alone
        start = rng.choice([0, 0, BLOCK * rng.randint(1, 127)])
        return dict(kind=kind, model=name, layers=layers, batch=0, k=0, lo=0, hi=0, shared=0, piece=_spread(rng, 9, 1400), start=start)
    batch = _spread(rng, 1, 64)
    k = 0 if kind == "decode" else rng.randint(0, 6)
    hi = _spread(rng, 40, min(6000, tokens // batch))
    lo = max(1, hi // rng.choice([1, 2, 4]))
    shared = BLOCK * rng.randint(1, max(1, lo // BLOCK // 2)) if batch > 1 and lo > 4 * BLOCK and rng.random() < 0.25 else 0
    piece = _spread(rng, 9, 700) if kind == "forward" and rng.random() < 0.4 else 0
    return dict(kind=kind, model=name, layers=layers, batch=batch, k=k, lo=lo, hi=hi, shared=shared, piece=piece, start=0)


# ---- what a program has in hand -----------------------------------------------------------------------------------

_context = None


def _ctx():
    """The process's one context: a program opens one for each GPU and keeps it."""
    global _context
    if _context is None:
        _context = api.Context(0)
    return _context


def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _quantised(rows, cols, bits, group, std, g):
    """N(0, std) weights in the mlx layout, made some rows at a time."""
    per, parts = max(1, (1 << 26) // cols), []
    for r in range(0, rows, per):
        w = torch.empty(min(per, rows - r), cols, device="cuda").normal_(0.0, std, generator=g)
        parts.append(quantize_affine(w, bits, group))
    return [torch.cat(t) if len(parts) > 1 else t[0] for t in zip(*parts)]


def _load(case, seed, seqs):
    """A model with random layers whose greedy choice after token t is follow[t]."""
    cfg = truncated(PRESETS[case["model"]], case["layers"])
    g = _generator(seed, 1)
    ck = synth_checkpoint(cfg, seed=int(seed), device="cuda", std=0.01)
    hidden, vocab = cfg.hidden_size, cfg.vocab_size
    gemma = cfg.model_type == "gemma2"           # its embedding is scaled by sqrt(hidden) on the way in
    w, s, b = _quantised(vocab, hidden, cfg.bits, cfg.group_size, 2.0 * hidden ** -0.5 if gemma else 2.0, g)
    ck["model.embed_tokens.weight"], ck["model.embed_tokens.scales"], ck["model.embed_tokens.biases"] = w, s, b
    if gemma:                                    # its sublayers are normalised on the way out: the same tenth
        for name, t in ck.items():
            if name.endswith("post_attention_layernorm.weight") or name.endswith("post_feedforward_layernorm.weight"):
                t.fill_(-0.8)
    if cfg.tie_word_embeddings:
        follow = torch.arange(vocab, device="cuda")
        if not gemma:                            # logits of a few units, not of a few hundred
            ck["model.norm.weight"].fill_(0.01)
    else:
        before = torch.randperm(vocab, device="cuda", generator=g)
        follow = torch.empty_like(before)
        follow[before] = torch.arange(vocab, device="cuda")
        ck["lm_head.weight"], ck["lm_head.scales"], ck["lm_head.biases"] = w[before], s[before] * 0.01, b[before] * 0.01
    model = api.CudaModel(_ctx(), cfg, ck, max_step_tokens=CHUNK, max_step_seqs=max(64, seqs))
    return cfg, model, follow.cpu().numpy()


def _lengths(case, rng):
    """Tokens in the cache of each sequence before the call: one at each end of the range, the others between."""
    n = rng.integers(case["lo"], case["hi"] + 1, size=case["batch"])
    if case["batch"] >= 2:
        n[0], n[1] = case["lo"], case["hi"]
    return [int(v) for v in n]


def _fill(model, kv, prompt, blocks):
    """Runs a prompt through the model, chunk by chunk."""
    for at in range(0, len(prompt), CHUNK):
        ids = prompt[at: at + CHUNK]
        model.forward_step(api.StepBatch(ids, [api.SeqStep(len(ids), at, 0, blocks)]), kv)


def _prepare_model(case, seed):
    rng = np.random.default_rng(int(seed))
    cfg, model, follow = _load(case, seed, case["batch"] + 1)
    lens, rows = _lengths(case, rng), case["k"] + 1
    need = [-(-(n + rows + 1) // BLOCK) for n in lens]           # one slot more: a decode pass takes two steps
    shared = case["shared"] // BLOCK
    piece, start = case["piece"], case["start"]
    first = -(-max(lens + [start + piece]) // BLOCK)             # blocks 0 .. first - 1: the prompt that the others copy
    total = first + sum(n - shared for n in need) + -(-(start + piece) // BLOCK)
    kv = api.PagedKv(_ctx(), model.kv_spec(total, BLOCK))
    prompt = rng.integers(0, cfg.vocab_size, max(lens + [start])).astype(np.uint32)
    if len(prompt):
        _fill(model, kv, prompt, np.arange(first, dtype=np.uint32))
    # a running server's free list is in no order
    free = iter(rng.permutation(np.arange(first, total)).astype(np.uint32))
    seqs, ids, drafts = [], [], []
    for n, blocks in zip(lens, need):
        own = np.array([next(free) for _ in range(blocks - shared)], dtype=np.uint32)
        for j in range(shared, -(-n // BLOCK)):
            kv.copy_block(j, int(own[j - shared]))
        table = np.concatenate([np.arange(shared, dtype=np.uint32), own])
        t = int(rng.integers(cfg.vocab_size))
        row = [t]
        for _ in range(case["k"]):
            t = int(follow[t]) if rng.random() < ACCEPT else int(rng.integers(cfg.vocab_size))
            row.append(t)
        ids += row
        seqs.append(api.SeqStep(rows, n, rows, table))
    if piece:
        table = np.array([next(free) for _ in range(-(-(start + piece) // BLOCK))], dtype=np.uint32)
        for j in range(-(-start // BLOCK)):
            kv.copy_block(j, int(table[j]))
        ids += [int(v) for v in rng.integers(0, cfg.vocab_size, piece)]
        seqs.append(api.SeqStep(piece, start, 1, table))
    state = {"kind": case["kind"], "model": model, "kv": kv}
    if case["kind"] == "draft":
        model.set_stream_lane(True)
        state.update(first=ids[0], offset=lens[0], blocks=seqs[0].blocks, k=case["k"])
    elif case["kind"] == "decode":
        later = [api.SeqStep(1, s.offset + 1, 1, s.blocks) for s in seqs]
        state.update(one=api.StepBatch(np.array(ids, dtype=np.uint32), seqs), two=api.StepBatch(np.zeros(len(ids), dtype=np.uint32), later),
                     host=np.full(len(ids), -1, dtype=np.int32), fed=np.arange(len(ids), dtype=np.int32))
    else:
        state.update(batch=api.StepBatch(np.array(ids, dtype=np.uint32), seqs))
    _ctx().sync()
    return state


def _prepare_linear(case, seed):
    g = _generator(seed, 2)
    w, s, b = _quantised(case["n_out"], case["n_in"], case["bits"], case["group"], 0.02, g)
    weight = api.QuantizedWeight(_ctx(), w, s, b, case["bits"], case["group"])
    x = torch.empty(case["rows"], case["n_in"], device="cuda").normal_(generator=g).to(torch.bfloat16)
    return {"kind": "linear", "weight": weight, "x": x}


def _prepare_attention(case, seed):
    rng = np.random.default_rng(int(seed))
    g = _generator(seed, 3)
    lens, rows = _lengths(case, rng), case["k"] + 1
    need = [-(-(n + rows) // BLOCK) for n in lens]
    kv = api.PagedKv(_ctx(), api.KvSpec(1, case["kv_heads"], case["head_dim"], sum(need) + 64, BLOCK))
    block = kv.bytes_per_block() // 2
    for j in range(64):                                          # 64 blocks of random content, copied over the pool
        data = torch.empty(block, device="cuda").normal_(generator=g).to(torch.bfloat16)
        kv.write_block_bytes(j, data.view(torch.uint8).cpu().numpy().tobytes())
    order = rng.permutation(np.arange(64, sum(need) + 64)).astype(np.uint32)
    for j in order:
        kv.copy_block(int(rng.integers(64)), int(j))
    seqs, at = [], 0
    for n, blocks in zip(lens, need):
        seqs.append(api.SeqStep(rows, n, rows, order[at: at + blocks]))
        at += blocks
    q = torch.empty(rows * len(lens), case["heads"], case["head_dim"], device="cuda").normal_(generator=g).to(torch.bfloat16)
    _ctx().sync()
    return {"kind": "attention", "kv": kv, "q": q, "seqs": seqs, "scale": case["head_dim"] ** -0.5}


def prepare(case, seed):
    if case["kind"] == "linear":
        return _prepare_linear(case, seed)
    if case["kind"] == "attention":
        return _prepare_attention(case, seed)
    return _prepare_model(case, seed)


# ---- one pass -----------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "verify":
        return state["model"].verify_step(state["batch"], state["kv"])
    if kind == "forward":
        logits = state["model"].forward_step(state["batch"], state["kv"])
        logits.owner = state["model"]   # the tensor is the model's own buffer: it must not outlive the model
        return logits
    if kind == "decode":
        m, kv, n = state["model"], state["kv"], len(state["host"])
        a = m.decode_launch(state["one"], kv, state["host"])
        b = m.decode_launch(state["two"], kv, state["fed"])
        return [np.array(m.decode_collect(a, n)), np.array(m.decode_collect(b, n))]
    if kind == "draft":
        return np.array(state["model"].draft_chain(state["kv"], state["first"], state["offset"], state["blocks"], state["k"]))
    if kind == "linear":
        return state["weight"].matmul(state["x"])
    return api.paged_attention(_ctx(), state["kv"], 0, state["q"], state["seqs"], state["scale"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def _weight_bytes(n_out, n_in, bits, group):
    return n_out * n_in * bits / 8 + 2 * n_out * (n_in // group) * 2


def work(case):
    if case["kind"] == "linear":
        m, n, k = case["rows"], case["n_out"], case["n_in"]
        return {"bytes": _weight_bytes(n, k, case["bits"], case["group"]) + 2.0 * m * (n + k), "flops": 2.0 * m * n * k}
    rows, mean = case["k"] + 1, (case["lo"] + case["hi"]) / 2
    if case["kind"] == "attention":
        per = 4 * case["kv_heads"] * case["head_dim"]
        q = case["batch"] * rows * case["heads"] * case["head_dim"]
        return {"bytes": case["batch"] * (mean + rows) * per + 4.0 * q, "flops": 4.0 * q * (mean + rows / 2)}
    c, layers = PRESETS[case["model"]], case["layers"]
    h, d, f, v = c.hidden_size, c.head_dim, c.intermediate_size, c.vocab_size
    qd, kd = c.num_attention_heads * d, c.num_key_value_heads * d
    linears = [(qd + 2 * kd, h), (h, qd), (2 * f, h), (h, f)]
    layer_bytes = sum(_weight_bytes(n, k, c.bits, c.group_size) for n, k in linears)
    layer_ops = sum(n * k for n, k in linears)
    head = _weight_bytes(v, h, c.bits, c.group_size)
    kv_token = layers * 4 * kd                                  # K and V of one position
    if case["kind"] == "draft":                                 # k forwards of one row, one after the other
        k = case["k"]
        return {"bytes": k * (layers * layer_bytes + head + (mean + k / 2) * kv_token), "flops": 2.0 * k * (layers * (layer_ops + 2 * qd * mean) + v * h)}
    shared = case["shared"] if case["batch"] else 0
    own = case["batch"] * (mean - shared) + shared              # cached positions, the shared ones once
    m = case["batch"] * rows + case["piece"]
    sampled = case["batch"] * rows + (1 if case["piece"] else 0)
    pairs = case["batch"] * rows * (mean + rows / 2) + case["piece"] * (case["start"] + case["piece"] / 2)
    if c.sliding_window:                                        # every second layer sees the last keys only
        seen = min(1.0, c.sliding_window / max(1.0, mean))
        own, pairs = own * (1 + seen) / 2, pairs * (1 + seen) / 2
    out = sampled * v * 2 if case["kind"] == "forward" else 0   # the logits, where they are what comes back
    one = {"bytes": layers * layer_bytes + head + (own + case["start"] + m) * kv_token + out,
           "flops": 2.0 * m * layers * layer_ops + 2.0 * sampled * v * h + 4.0 * pairs * qd * layers}
    times = 2 if case["kind"] == "decode" else 1                # a decode pass is two steps
    return {n: times * b for n, b in one.items()}


def tolerance(case):
    # Tokens and counts: nearly every next token has a clear winner (above), so few change with the rounding of a sum.
    if case["kind"] in ("verify", "decode", "draft"):
        return {"differ": 0.01}
    # One bf16 result of fp32 sums over bf16 operands.
    if case["kind"] in ("linear", "attention"):
        return {"rel": 6e-3}
    # bf16 logits of a whole model: each layer rounds its activations to bf16 about eight times (2^-9 each), and sums in
    # another order make other roundings. Measured with the sums along K cut in other places: 1.3e-2 at 32 layers.
    return {"rel": 4e-3 * PRESETS[case["model"]].num_hidden_layers ** 0.5}
