"""What this library is timed on: single-sequence and batched decoding, prompt ingestion and the stand-alone quantised
product, over the model shapes, formats, batch widths and context lengths that bench.py and the tests configure.

A program keeps one loaded model and serves one request after the other with it, so a model is loaded once per process
and format (`_engine`); what a case prepares is the requests: their prompts, the key/value pages these leave behind, the
tokens of the next step. Every state has its own sequences (slots and scattered pages) in the model's pool and gives them
back when it is dropped.

The weights are random blocks with the statistics of a trained model in three respects: zero mean, a residual stream in
which each layer adds a fraction of what is there, and an output matrix that scores a plausible successor of the current
token well above the rest (the output row of token (t + 1) is the embedding row of t; with tied embeddings, its own). So
the greedy token does not hang on the last bits of a logit, as it would with independent random matrices."""
import math
import random
import weakref
from collections import OrderedDict

import numpy as np
import torch

import jitllm_b200 as jl
from jitllm_b200 import GGMLType, TensorRole

# dim, hidden, layers, heads, kv heads, vocabulary, context, tied embeddings: the shapes bench.py decodes with. The 8B
# context holds the longest prompt of its prefill sweep and the tokens after it.
ARCHS = {
    "tiny": (512, 1024, 4, 8, 2, 4096, 1024, False),
    "1b": (2048, 8192, 16, 32, 8, 128256, 2048, True),
    "8b": (4096, 14336, 32, 32, 8, 128256, 8448, False),
}
PAGE = 16            # tokens per page
MAX_BATCH = 64
STATE_TOKENS = 32768  # context tokens that one state's sequences hold together
STATES = 5           # states of one model that are alive at once
ENGINES = 4          # models that stay loaded


def listed():
    return [
        # one token of a small model, logits to a host sampler: latency and launches only
        {"name": "tiny q4_0 step", "kind": "decode", "arch": "tiny", "format": "Q4_0", "batch": 1, "context": 57, "idle": 0, "out": "logits"},
        # single-sequence greedy decoding right after a short prompt
        {"name": "1b q8_0 generate 32", "kind": "generate", "arch": "1b", "format": "Q8_0", "batch": 1, "context": 32, "idle": 0, "steps": 32},
        # chat with a short history, tokens fed back on the device
        {"name": "8b q4_k generate 16", "kind": "generate", "arch": "8b", "format": "Q4_K", "batch": 1, "context": 512, "idle": 0, "steps": 16},
        # a mixed-precision file and a long history, logits to a host sampler
        {"name": "8b mixed step at 3901", "kind": "decode", "arch": "8b", "format": "mixed", "batch": 1, "context": 3901, "idle": 0, "out": "logits"},
        # a small server batch, sequences of different lengths, one slot free, logits to host samplers
        {"name": "8b q4_k batch 8 logits", "kind": "decode", "arch": "8b", "format": "Q4_K", "batch": 8, "context": 700, "idle": 1, "out": "logits"},
        # a server batch, greedy
        {"name": "8b q4_k batch 32", "kind": "decode", "arch": "8b", "format": "Q4_K", "batch": 32, "context": 512, "idle": 0, "out": "greedy"},
        # the widest batch, temperature / top-p sampling on the device
        {"name": "8b q8_0 batch 64 sampled", "kind": "decode", "arch": "8b", "format": "Q8_0", "batch": 64, "context": 420, "idle": 0, "out": "sampled"},
        # time to the first token: a one-line question, an ordinary prompt, the longest one
        {"name": "1b q8_0 prompt 23", "kind": "prompt", "arch": "1b", "format": "Q8_0", "tokens": 23, "start": 0},
        {"name": "8b q4_k prompt 471", "kind": "prompt", "arch": "8b", "format": "Q4_K", "tokens": 471, "start": 0},
        {"name": "8b q8_0 prompt 8192", "kind": "prompt", "arch": "8b", "format": "Q8_0", "tokens": 8192, "start": 0},
        # the stand-alone product: one attention projection by one vector, one feed-forward matrix by a block of rows
        {"name": "q4_0 4096x4096 n1", "kind": "product", "format": "Q4_0", "rows": 4096, "cols": 4096, "n": 1},
        {"name": "q4_k 14336x4096 n512", "kind": "product", "format": "Q4_K", "rows": 14336, "cols": 4096, "n": 512},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "generate", "prompt", "prompt", "product"])
    if kind == "product":
        rows, cols = _log_int(rng, 256, 128256), 256 * _log_int(rng, 2, 56)
        most = max(1, int(1e13 / (rows * cols)))
        return {"kind": kind, "format": rng.choice(["Q8_0", "Q4_0", "Q4_K", "Q8_0", "Q4_0", "Q4_K", "Q6_K", "Q5_K", "Q4_1"]), "rows": rows, "cols": cols,
                "n": _log_int(rng, 1, min(2048, most))}
    arch = rng.choice(["tiny", "1b", "8b", "8b"])
    case = {"kind": kind, "arch": arch, "format": rng.choice(["Q4_K", "Q8_0", "Q4_0", "mixed"] if arch == "8b" else ["Q4_K", "Q8_0", "Q4_0"])}
    longest = ARCHS[arch][6] - 160
    if kind == "prompt":
        tokens = _log_int(rng, 2, min(longest, 8000))
        start = rng.choice([0, 0, PAGE * rng.randrange(1, 40)])  # behind a system prompt that is there already
        case.update(tokens=tokens, start=start if tokens + start <= longest else 0)
        return case
    batch = rng.choice([1, 1, _log_int(rng, 2, MAX_BATCH)])
    # the longest row of a batch holds 1.5 times the nominal context
    context = _log_int(rng, 8, min(4096, int(longest / 1.5), STATE_TOKENS // batch))
    case.update(batch=batch, context=context, idle=rng.randrange(0, 1 + batch // 4))
    if kind == "generate":
        case["steps"] = _log_int(rng, 4, 32)
    else:
        case["out"] = rng.choice(["greedy", "logits", "sampled"])
    return case


# ------------------------------------------------------------------------------------------------ weights

def _blocks(kind, elements, std, gen):
    """[blocks, bytes] on the GPU: random quantised blocks of zero-mean weights of this standard deviation."""
    t = GGMLType[kind]
    n = elements // t.block_size
    raw = torch.randint(0, 256, (n, t.type_size), dtype=torch.uint8, device="cuda", generator=gen)
    # (bytes of the scale, standard deviation of code times sub-scale, mean code of the formats with a minimum)
    unit = {"Q4_0": 4.61, "Q4_1": 4.61, "Q8_0": 73.9, "Q4_K": 4.61 * 48, "Q5_K": 9.23 * 48, "Q6_K": 18.5 * 73.9}[kind]
    d = (torch.rand(n, device="cuda", generator=gen) * 0.6 + 0.7) * (std / unit)
    if kind in ("Q4_0", "Q8_0", "Q6_K"):
        d = d * (torch.randint(0, 2, (n,), device="cuda", generator=gen) * 2 - 1)
    d = d.to(torch.float16)
    at = 208 if kind == "Q6_K" else 0
    raw[:, at:at + 2] = d.view(torch.uint8).view(n, 2)
    mean = {"Q4_1": -7.5, "Q4_K": 7.5, "Q5_K": 15.5}.get(kind)
    if mean is not None:
        raw[:, 2:4] = (d * mean).to(torch.float16).view(torch.uint8).view(n, 2)
    if kind in ("Q4_K", "Q5_K"):  # eight 6-bit scales between 32 and 63, minima equal to them
        raw[:, 4:8] |= 0xA0
        raw[:, 8:12] = raw[:, 4:8]
        raw[:, 12:16] &= 0x0F
        raw[:, 12:16] |= raw[:, 12:16] << 4
    return raw


def _host(raw):
    out = torch.empty(raw.shape, dtype=torch.uint8, pin_memory=True)
    out.copy_(raw)
    return out.numpy().reshape(-1)


class _Engine:
    """One loaded model with its page pool."""

    def __init__(self, arch, fmt):
        dim, hidden, layers, heads, kv_heads, vocab, ctx, tied = ARCHS[arch]
        self.config = c = jl.Configuration(dim, hidden, layers, heads, kv_heads, vocab, ctx, tiedEmbeddings=tied)
        self.dev = jl.Device(0)
        self.model = m = jl.B200Model(self.dev, c, maxBatch=MAX_BATCH)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(20261125)
        base = "Q4_K" if fmt == "mixed" else fmt

        def matrix(role, layer, kind, std=0.02):
            rows, cols = c.matrix_shape(role)
            raw = _blocks(kind, rows * cols, std, gen)
            m.uploadTensor(role, layer, GGMLType[kind], _host(raw))
            return raw

        def norm(role, layer, size):
            w = (torch.rand(dim, device="cuda", generator=gen) * 0.4 + 0.8) * size
            m.uploadTensor(role, layer, GGMLType.F32, w.cpu().numpy())

        top = "Q6_K" if fmt == "mixed" else base
        table = matrix(TensorRole.TOKEN_EMBEDDING, -1, top, 1.0)
        for l in range(layers):
            # mixed-precision files keep the value and down projections of half of the layers in more bits
            more = "Q6_K" if fmt == "mixed" and l % 2 == 0 else base
            norm(TensorRole.ATTENTION_NORM, l, 0.5)
            matrix(TensorRole.ATTENTION_QUERY, l, base)
            matrix(TensorRole.ATTENTION_KEY, l, base)
            matrix(TensorRole.ATTENTION_VALUE, l, more)
            matrix(TensorRole.ATTENTION_OUTPUT, l, base)
            norm(TensorRole.FFN_NORM, l, 0.35)
            matrix(TensorRole.FFN_GATE, l, base)
            matrix(TensorRole.FFN_UP, l, base)
            matrix(TensorRole.FFN_DOWN, l, more)
        norm(TensorRole.OUTPUT_NORM, -1, 1.4 / math.sqrt(dim))  # logits of a standard deviation between 1 and 2
        if not tied:
            m.uploadTensor(TensorRole.OUTPUT, -1, GGMLType[top], _host(torch.roll(table.view(vocab, -1), 1, 0)))
        del table
        m.uploadRope(*jl.precomputeFreqsCis(ctx, c.headSize, c.ropeTheta))
        m.finalize()
        self.per_slot = (ctx + PAGE - 1) // PAGE
        slots = MAX_BATCH * STATES
        pages = min(STATE_TOKENS * 5 // 4 // PAGE, MAX_BATCH * self.per_slot) * STATES
        self.kv = m.createKvStorage(jl.KvStorageRequest(pages, self.per_slot, slots, PAGE, layers, c.kvDim))
        self.table = np.full((slots, self.per_slot), jl.UNMAPPED, dtype=np.int32)
        self.free_slots = list(range(slots))[::-1]
        self.free_pages = list(range(pages))
        random.Random(7).shuffle(self.free_pages)
        self.executor = jl.B200BatchExecutor(m)


_engines = OrderedDict()


def _engine(arch, fmt):
    key = (arch, fmt)
    if key not in _engines:
        while len(_engines) >= ENGINES:
            _engines.popitem(last=False)
        _engines[key] = _Engine(arch, fmt)
    _engines.move_to_end(key)
    return _engines[key]


class _Sequences:
    """Slots with room for so many tokens each, leased from a model's pool for as long as this object lives."""

    def __init__(self, engine, lengths):
        self.slots, self.pages = [], []
        for n in lengths:
            slot = engine.free_slots.pop()
            need = (n + PAGE - 1) // PAGE
            pages = [engine.free_pages.pop() for _ in range(need)]
            engine.table[slot, :need] = pages
            self.slots.append(slot)
            self.pages += pages
        engine.kv.publishBlockTable(engine.table.reshape(-1))
        weakref.finalize(self, self.give_back, engine, self.slots, self.pages)

    @staticmethod
    def give_back(engine, slots, pages):
        engine.table[slots] = jl.UNMAPPED
        engine.free_slots += slots
        engine.free_pages += pages


# ------------------------------------------------------------------------------------------------ states

def _contexts(case):
    """Tokens in front of the next one, row by row: half to one and a half times the nominal context of a batch."""
    b = case["batch"]
    if b == 1:
        return [case["context"]]
    return [max(1, int(case["context"] * (0.5 + i / (b - 1)))) for i in range(b)]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    rng = np.random.default_rng(seed)
    if case["kind"] == "product":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        rows, cols, n = case["rows"], case["cols"], case["n"]
        s.engine = _device()
        s.matrix = s.engine.upload_matrix(GGMLType[case["format"]], _host(_blocks(case["format"], rows * cols, 0.02, gen)), rows, cols)
        s.x = torch.randn((n, cols), device="cuda", generator=gen)
        s.y = torch.empty((n, rows), device="cuda")
        torch.cuda.synchronize()
        return s
    s.engine = e = _engine(case["arch"], case["format"])
    vocab = e.config.vocabularySize
    if case["kind"] == "prompt":
        start, n = case["start"], case["tokens"]
        s.sequences = _Sequences(e, [start + n])
        s.boundary = jl.B200InvocationBoundary(e.model, kvSlot=s.sequences.slots[0])
        s.prompt = rng.integers(0, vocab, start + n).astype(np.int32)
        if start:
            s.boundary.prefill(s.prompt[:start])
        s.prompt = s.prompt[start:]
        return s
    lengths = _contexts(case)
    steps = case.get("steps", 1)
    s.sequences = _Sequences(e, [n + steps for n in lengths])
    active = [i < case["batch"] - case["idle"] for i in range(case["batch"])]
    for slot, n, on in zip(s.sequences.slots, lengths, active):
        if on:
            jl.B200InvocationBoundary(e.model, kvSlot=slot).prefill(rng.integers(0, vocab, n).astype(np.int32))
    s.batch = jl.BatchSlots(active, [int(t) for t in rng.integers(0, vocab, case["batch"])], lengths, s.sequences.slots)
    s.sampler = jl.Sampler.selectSampler(vocab, 0.8, 0.9, seed) if case.get("out") == "sampled" else None
    return s


_dev = None


def _device():
    global _dev
    if _dev is None:
        _dev = jl.Device(0)
    return _dev


def run(s):
    case, e = s.case, s.engine
    if case["kind"] == "product":
        s.matrix.matmul_dev(s.x.data_ptr(), case["n"], s.y.data_ptr())
        return s.y
    if case["kind"] == "prompt":
        # the prompt but for its last token, then the step that scores the first new one
        s.boundary.prefill(s.prompt[:-1], case["start"])
        r = s.boundary.invoke(int(s.prompt[-1]), case["start"] + case["tokens"] - 1)
        return {"logits": r.logits, "token": r.sampledToken}
    if case["kind"] == "generate":
        return e.executor.generate(s.batch, case["steps"])
    if case["out"] == "logits":
        tokens, logits = e.executor.decodeStep(s.batch, wantLogits=True)
        return {"logits": logits[np.asarray(s.batch.active)], "tokens": tokens}
    return e.executor.decodeStep(s.batch, sampler=s.sampler)


# ------------------------------------------------------------------------------------------------ accounting

def _model_bytes(arch, fmt, head):
    """(bytes, weights) that one step reads of the layers' matrices, and of the output matrix where `head`."""
    dim, hidden, layers, heads, kv_heads, vocab, _, tied = ARCHS[arch]
    kv = dim * kv_heads // heads
    base = GGMLType["Q4_K" if fmt == "mixed" else fmt]
    total, weights = 0, 0
    for l in range(layers):
        more = GGMLType.Q6_K if fmt == "mixed" and l % 2 == 0 else base
        for t, n in ((base, dim * (2 * dim + kv + 2 * hidden)), (more, dim * (kv + hidden))):
            total += t.byte_size_for(n)
            weights += n
    if head:
        total += (GGMLType.Q6_K if fmt == "mixed" else base).byte_size_for(vocab * dim)
        weights += vocab * dim
    return total, weights


def work(case):
    if case["kind"] == "product":
        rows, cols, n = case["rows"], case["cols"], case["n"]
        return {"bytes": GGMLType[case["format"]].byte_size_for(rows * cols) + 4 * n * (rows + cols), "flops": 2 * rows * cols * n}
    dim, hidden, layers, heads, kv_heads, vocab, _, _ = ARCHS[case["arch"]]
    kv_token = 2 * 2 * layers * (dim * kv_heads // heads)
    layer_bytes, layer_weights = _model_bytes(case["arch"], case["format"], False)
    step_bytes, step_weights = _model_bytes(case["arch"], case["format"], True)
    if case["kind"] == "prompt":
        n, start = case["tokens"], case["start"]
        keys = sum(range(start + 1, start + n + 1))
        # the prompt's keys and values are written once; the last token's step reads every key and value and the weights
        return {"bytes": (layer_bytes if n > 1 else 0) + step_bytes + (start + 2 * n) * kv_token + 4 * vocab,
                "flops": 2 * layer_weights * (n - 1) + 2 * step_weights + 4 * dim * layers * keys}
    steps = case.get("steps", 1)
    rows = [n for i, n in enumerate(_contexts(case)) if i < case["batch"] - case["idle"]]
    keys = sum(n + k + 1 for n in rows for k in range(steps))
    out = 4 * vocab * len(rows) if case.get("out") == "logits" else 0
    return {"bytes": steps * step_bytes + keys * kv_token + out,
            "flops": 2 * step_weights * len(rows) * steps + 4 * dim * layers * keys}


def tolerance(case):
    # a product: activations of 16 bits per block of 32, or weights rounded to binary16 (2^-11 each); the logits: that,
    # binary16 keys and values, and the depth of the model
    return {"rel": 1e-3} if case["kind"] == "product" else {"rel": 1e-2}
