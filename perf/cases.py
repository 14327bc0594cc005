"""The work this package does for its users, as cases that can be timed: linears over compressed weights, whole decoder
steps, indexed decoding of frames on the GPU and the host codec that makes and reads the frames.

Ranges.  Linears: batches of 1 to 768 rows over the four linears of a decoder layer (the benchmark's shapes, their
tensor-parallel shards, and a 4096-wide layer), and single ragged linears of a hundred to four thousand rows and
columns.  Steps: 1 to 128 sequences with 128 to 2048 tokens of context, verify passes of 2 to 128 rows, prompts of 16 to
1000 tokens.  Frames: 256 x 256 to 4096 x 4096 words on the GPU, up to 1024 x 2048 on the host.  Everything is BF16 with the
package's default layout, which is what a user gets who asks for nothing else.
"""
import math

import numpy as np
import torch

from georefine_b200 import codec, serve
from georefine_b200.gpu import CudaContextTensor
from georefine_b200.resident import ResidentWeight
from georefine_b200.serving import BctxEmbedding, BctxLinear

DEVICE = "cuda:0"
HEADS, KV_HEADS, HEAD_DIM, HIDDEN, FFN = 40, 8, 128, 5120, 17408   # the benchmark's decoder
LAYERS, VOCAB = 4, 9504   # its stack of 64 layers and 152064 tokens, depth and vocabulary cut by 16 together
# hidden, query heads, KV heads, FFN width of a layer as one GPU holds it: whole, its 2- and 4-way shards, a smaller model
LAYER_SHAPES = ((5120, 40, 8, 17408), (5120, 20, 4, 8704), (5120, 10, 2, 4352), (4096, 32, 8, 14336))


def listed():
    layer = {"op": "layer", "hidden": HIDDEN, "heads": HEADS, "kv_heads": KV_HEADS, "ffn": FFN}
    return [
        # one nn.Linear replacement with a bias on a handful of rows, ragged in every dimension: latency of a call
        {"name": "linear_ragged", "op": "linear", "rows": 777, "cols": 1032, "m": 6, "bias": True},
        # the four linears of a layer when one sequence is decoded: weight streaming
        {"name": "layer_m1", "m": 1, **layer},
        # the same at full continuous batching, and in the verify pass of 128 sequences with 5 drafts each
        {"name": "layer_m128", "m": 128, **layer},
        {"name": "layer_m768", "m": 768, **layer},
        # the whole decode step of one interactive sequence, and of a full batch, with 2048 tokens of context
        {"name": "step_1", "op": "step", "seqs": 1, "context": 2048},
        {"name": "step_128", "op": "step", "seqs": 128, "context": 2048},
        # a speculative verify pass: 16 sequences, the pending token and 5 drafts each
        {"name": "verify_16x6", "op": "verify", "seqs": 16, "drafts": 5, "context": 1024},
        # a prompt taken in through the session, in the session's own chunks of rows
        {"name": "prefill_1000", "op": "prefill", "tokens": 1000},
        # a weight decoded densely from its unchanged frame (`.weight` of a compressed linear), the one-matrix benchmark
        {"name": "frame_decode", "op": "frame_decode", "rows": 4096, "cols": 4096},
        # embedding rows for a batch of tokens, decoded from a compressed table
        {"name": "embedding_128", "op": "embedding", "rows": 2048, "cols": 5120, "ids": 128},
        # packaging a checkpoint's tensor on the host, and reading one back
        {"name": "host_encode", "op": "host_encode", "rows": 1024, "cols": 2048},
        {"name": "host_decode", "op": "host_decode", "rows": 1024, "cols": 2048},
    ]


def _spread(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(("linear", "layer", "layer", "step", "step", "verify", "prefill", "frame_decode", "embedding", "host_encode", "host_decode"))
    if op == "linear":
        return {"op": op, "rows": _spread(rng, 128, 4096), "cols": _spread(rng, 128, 4096), "m": _spread(rng, 1, 64), "bias": rng.random() < 0.5}
    if op == "layer":
        hidden, heads, kv_heads, ffn = rng.choice(LAYER_SHAPES)
        return {"op": op, "hidden": hidden, "heads": heads, "kv_heads": kv_heads, "ffn": ffn, "m": _spread(rng, 1, 768)}
    if op == "step":
        return {"op": op, "seqs": _spread(rng, 1, 128), "context": _spread(rng, 128, 2048)}
    if op == "verify":
        drafts = rng.randint(1, 5)
        return {"op": op, "seqs": _spread(rng, 1, 128 // (drafts + 1)), "drafts": drafts, "context": _spread(rng, 128, 2048)}
    if op == "prefill":
        return {"op": op, "tokens": _spread(rng, 16, 1000)}
    if op == "embedding":
        # widths of embedding tables are multiples of 128; now and then one that is not
        cols = 128 * _spread(rng, 4, 40) if rng.random() < 0.75 else _spread(rng, 512, 5120)
        return {"op": op, "rows": _spread(rng, 256, 2048), "cols": cols, "ids": _spread(rng, 1, 256)}
    if op == "frame_decode":
        return {"op": op, "rows": _spread(rng, 256, 4096), "cols": _spread(rng, 256, 4096)}
    return {"op": op, "rows": _spread(rng, 64, 1024), "cols": _spread(rng, 64, 2048)}


# ---- inputs ------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _words(rows, cols, g):
    """BF16 bit patterns of N(0, 0.02) weights with a LogNormal(0, 0.25) scale per row, on the host."""
    w = torch.randn(rows, cols, generator=g, device=DEVICE) * 0.02
    w *= torch.exp(0.25 * torch.randn(rows, 1, generator=g, device=DEVICE))
    return w.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


def _rows(m, cols, g):
    return torch.randn(m, cols, generator=g, device=DEVICE).to(torch.bfloat16)


def _resident(words):
    # a loader knows the digest of its words from the frame: it is not computed again here
    return ResidentWeight.from_words(words, DEVICE, source_sha256=bytes(32), verify=False)


def _layer_shapes(case):
    h, q, f = case["hidden"], case["heads"] * HEAD_DIM, case["ffn"]
    return ((q + 2 * case["kv_heads"] * HEAD_DIM, h), (h, q), (2 * f, h), (h, f))


def _decoder_weights(seed):
    cfg = serve.DecoderConfig(hidden=HIDDEN, layers=LAYERS, heads=HEADS, kv_heads=KV_HEADS, ffn=FFN, vocab=VOCAB)
    g = _generator(seed)
    shapes = {name: (n, k) for name, n, k in cfg.linear_shapes()}
    shapes.update(embed=(VOCAB, HIDDEN), lm_head=(VOCAB, HIDDEN))

    def words_of(name):
        leaf = name.split(".")[-1]
        if leaf in shapes:
            return _words(*shapes[leaf], g)
        scale = 1 + 0.1 * torch.randn(1, HIDDEN, generator=g, device=DEVICE)
        return scale.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)

    # one layer built on the host and copied on the device: the same bytes to stream for a fraction of the preparation
    return serve.DecoderWeights.from_words(cfg, words_of, DEVICE, distinct_layers=1, lin_factory=lambda name, words: _resident(words)), g


def _prepare_decoder(case, seed):
    """A decoder whose sequences already have their context in the KV cache, and the rows of the next step."""
    weights, g = _decoder_weights(seed)
    seqs, per = case["seqs"], case.get("drafts", 0) + 1
    n = seqs * per
    d = serve.BatchDecoder(weights, max_rows=max(n, 8), max_slots=seqs, max_context=case["context"] + 64, device=DEVICE)
    d.kv.normal_(generator=g)
    slots, positions = [], []
    for s in range(seqs):
        slot = d.open_slot()
        # sequences of a batch are not all equally long
        first = case["context"] - 1 - (s * 37) % max(1, case["context"] // 8)
        d.ensure_pages(slot, first + per)
        slots += [slot] * per
        positions += range(first, first + per)
    tokens = torch.randint(0, VOCAB, (n,), generator=g, device=DEVICE).tolist()
    return {"case": case, "decoder": d, "rows": (slots, positions, tokens), "n": n}


def prepare(case, seed):
    op = case["op"]
    g = _generator(seed)
    if op == "linear":
        frame = codec.encode(_words(case["rows"], case["cols"], g))
        bias = torch.nn.Parameter(_rows(1, case["rows"], g).reshape(-1), requires_grad=False) if case["bias"] else None
        return {"case": case, "module": BctxLinear(CudaContextTensor(frame, device=DEVICE), bias), "x": _rows(case["m"], case["cols"], g)}
    if op == "layer":
        m = case["m"]
        shapes = _layer_shapes(case)
        weights = [_resident(_words(n, k, g)) for n, k in shapes]
        weights[0].then(weights[1]).then(weights[2]).then(weights[3]).then(weights[0])
        return {"case": case, "weights": weights, "x": [_rows(m, k, g) for _, k in shapes],
                "y": [torch.empty(m, n, device=DEVICE, dtype=torch.bfloat16) for n, _ in shapes]}
    if op in ("step", "verify"):
        return _prepare_decoder(case, seed)
    if op == "prefill":
        weights, g = _decoder_weights(seed)
        session = serve.FastSession.load(weights=weights, device=DEVICE, max_len=1280)
        return {"case": case, "session": session, "ids": torch.randint(0, VOCAB, (case["tokens"],), generator=g, device=DEVICE).tolist()}
    words = _words(case["rows"], case["cols"], g)
    if op == "host_encode":
        return {"case": case, "words": words}
    frame = codec.encode(words)
    if op == "host_decode":
        return {"case": case, "frame": frame}
    tensor = CudaContextTensor(frame, device=DEVICE, fused=False)
    if op == "frame_decode":
        return {"case": case, "tensor": tensor}
    ids = torch.randint(0, case["rows"], (case["ids"],), generator=g, device=DEVICE)
    return {"case": case, "module": BctxEmbedding(tensor), "ids": ids}


# ---- one pass ----------------------------------------------------------------------------------------------------
def run(state):
    op = state["case"]["op"]
    if op == "linear":
        return state["module"](state["x"])
    if op == "layer":
        for w, x, y in zip(state["weights"], state["x"], state["y"]):
            w(x, y)
        return state["y"]
    if op in ("step", "verify"):
        d, n = state["decoder"], state["n"]
        d.set_rows(*state["rows"])
        d.run("ar" if op == "step" else "verify", n)
        return {"logits": d.logits[:n], "hidden": d.h[:n], "kv": d.kv}
    if op == "prefill":
        session = state["session"]
        st = session.prefill(token_ids=state["ids"])
        session.close(st)
        return {"logits": st.first_logits, "kv": session.d.kv}
    if op == "frame_decode":
        return state["tensor"].decode()
    if op == "embedding":
        return state["module"](state["ids"])
    if op == "host_encode":
        frame = codec.encode(state["words"])
        whole = np.zeros(codec.HEADER.size + 2 * state["words"].size + 32, dtype=np.uint8)   # no frame is longer than its words stored plainly
        whole[:len(frame)] = np.frombuffer(frame, dtype=np.uint8)
        return {"frame": whole, "bytes": len(frame)}
    return codec.decode(state["frame"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------
# Bytes of a weight in the form a pass reads it: the default resident layout (12 bits and a 0.4 % of bookkeeping), and a
# frame (6 bits stored raw and an exponent stream of about 4.5 bits).
RESIDENT, FRAME = 1.506, 1.31


def _decoder_work(rows, contexts):
    weights = LAYERS * sum(n * k for n, k in _layer_shapes({"hidden": HIDDEN, "heads": HEADS, "kv_heads": KV_HEADS, "ffn": FFN})) + VOCAB * HIDDEN
    kv = LAYERS * 2 * KV_HEADS * HEAD_DIM * 2 * sum(contexts)            # read once per sequence
    attention = LAYERS * 4 * HEADS * HEAD_DIM * sum(contexts) * (rows // len(contexts))
    return {"bytes": RESIDENT * weights + kv + rows * (HIDDEN + VOCAB) * 2, "flops": 2 * rows * weights + attention}


def work(case):
    op = case["op"]
    if op == "linear":
        n, k, m = case["rows"], case["cols"], case["m"]
        return {"bytes": RESIDENT * n * k + 2 * m * (n + k), "flops": 2 * m * n * k}
    if op == "layer":
        m = case["m"]
        return {"bytes": sum(RESIDENT * n * k + 2 * m * (n + k) for n, k in _layer_shapes(case)), "flops": 2 * m * sum(n * k for n, k in _layer_shapes(case))}
    if op in ("step", "verify"):
        return _decoder_work(case["seqs"] * (case.get("drafts", 0) + 1), [case["context"]] * case["seqs"])
    if op == "prefill":
        t = case["tokens"]
        w = _decoder_work(t, [t])
        w["flops"] -= 2 * (t - 1) * VOCAB * HIDDEN      # only the last position's logits are asked for
        w["flops"] -= LAYERS * 2 * HEADS * HEAD_DIM * t * (t - 1)   # a position attends to those before it
        w["bytes"] -= 2 * (t - 1) * VOCAB
        return w
    if op == "embedding":
        n = case["ids"] * case["cols"]
    else:
        n = case["rows"] * case["cols"]
    return {"bytes": (FRAME + 2) * n, "flops": 0}


def tolerance(case):
    op = case["op"]
    if op in ("linear", "layer"):
        return {"rel": 1e-2}       # one BF16 rounding of an FP32 sum
    if op in ("step", "verify", "prefill"):
        return {"rel": 2e-2}       # four layers, each with a dozen BF16 roundings on the way
    return "exact"                 # bit patterns and bytes
