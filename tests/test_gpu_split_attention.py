"""Decode attention with the keys split over CTAs, by itself: the attention output of a one-layer model's step against a 64-bit
softmax over the query, keys and values that the device itself used (the projections and pages are read back), at the depths
where the split changes: one key, around one tile of 64, where a second range, a third and the last of twenty (eight KV heads)
or thirty-seven (two) begin, where the fold takes another batch of ranges, and where ranges grow beyond a tile; every head size and group; queries of every magnitude; infinities and NaN among keys and values."""
import numpy as np
import pytest

import jitllm_b200 as jl
from jitllm_b200 import GGMLType, TensorRole
from tests.util import rel_l2

pytestmark = pytest.mark.gpu
# A score is a sum of head_dim exact products, added sixteen at a time into binary32: at most 8 + 3 additions cut off or rounded
# at 2^-23 of a partial sum of some 10, so 1e-5 of a weight in the worst case; outputs average the weights' errors.
BAR = 1e-5


def attention_outputs(dev, rope, heads, kv_heads, head, page, depths, width=1, std=0.05, seed=3, edit=None, special=None, token=5):
    """(output, 64-bit output, rotated query), [head][dimension] each, of one step at every depth (keys in the pages before it).
    `edit` changes the tensors, `special` the prompt ({position: token}), `token` is what row 0's step takes in."""
    cfg = jl.Configuration(dim=heads * head, hiddenDim=512, numberOfLayers=1, numberOfHeads=heads, numberOfKeyValueHeads=kv_heads,
                           vocabularySize=512, contextLength=max(depths) + 16)
    tensors = jl.synth_model_tensors(cfg, GGMLType.Q8_0, seed=seed, std=std)
    if edit is not None:
        edit(cfg, tensors)
    cr, ci = rope(cfg)
    model = jl.load_model(dev, cfg, tensors, cr, ci, maxBatch=width)
    bps = (cfg.contextLength + page - 1) // page
    kv = model.createKvStorage(jl.KvStorageRequest(width * bps, bps, width, page, 1, cfg.kvDim))
    kv.publishBlockTable(np.random.default_rng(seed).permutation(width * bps).astype(np.int32))
    kv.fill(0x7E00)  # NaN wherever nothing was written
    rng = np.random.default_rng(seed + 1)
    prompt = rng.integers(3, cfg.vocabularySize, size=max(depths)).astype(np.int32)
    for at, what in (special or {}).items():
        prompt[at] = what
    for b in range(width):
        jl.B200InvocationBoundary(model, kvSlot=b).prefill(prompt if max(depths) > 0 else [1], 0)
    ex = jl.B200BatchExecutor(model)
    cr, ci = np.asarray(cr, dtype=np.float32).reshape(-1, head // 2), np.asarray(ci, dtype=np.float32).reshape(-1, head // 2)
    out = []
    for pos in sorted(depths, reverse=True):  # the step overwrites the key at its position: deepest first
        rows = [max(0, pos - 3 * b) for b in range(width)]
        ex.decodeStep(jl.BatchSlots([True] * width, [token + b for b in range(width)], rows, list(range(width))))
        for b, p in enumerate(rows):
            q = model.debugRead("q", b).reshape(heads, head // 2, 2)
            q = np.stack([q[..., 0] * cr[p] - q[..., 1] * ci[p], q[..., 0] * ci[p] + q[..., 1] * cr[p]], axis=-1)
            q = q.reshape(heads, head).astype(np.float64)
            k, v = (np.stack([kv.readRow(w, b, 0, i).view(np.float16) for i in range(p + 1)]).astype(np.float64).reshape(p + 1, kv_heads, head)
                    for w in ("k", "v"))
            got = model.debugRead("xb", b).reshape(heads, head)
            want = np.empty((heads, head))
            with np.errstate(invalid="ignore"):
                for h in range(heads):
                    s = k[:, h * kv_heads // heads] @ q[h] / np.sqrt(head)
                    w = np.exp(s - s.max())
                    want[h] = (w / w.sum()) @ v[:, h * kv_heads // heads]
            out.append((got, want, q))
    kv.close()
    return out


def attention_errors(*args, **kwargs):
    """rel-L2 of the attention outputs of one step at every depth."""
    return [rel_l2(got.reshape(-1), want.reshape(-1)) for got, want, _ in attention_outputs(*args, **kwargs)]


def _rope(cfg):
    return jl.precomputeFreqsCis(cfg.contextLength, cfg.headSize, cfg.ropeTheta)


def _blocks(tensors, role, cols, layer=0):
    """Writable views of a Q8_0 matrix: the blocks' scales [row][block] and codes [row][block][32]."""
    t, raw = tensors[(role, layer)]
    tensors[(role, layer)] = (t, raw.copy())
    b = tensors[(role, layer)][1].view(np.dtype([("d", np.float16), ("q", np.int8, 32)])).reshape(-1, cols // 32)
    return b["d"], b["q"]


def _scaled(query, key, heads=slice(None)):
    """Query rows of these heads, and all key rows, times a power of two."""
    def edit(cfg, tensors):
        d, _ = _blocks(tensors, TensorRole.ATTENTION_QUERY, cfg.dim)
        rows = d.reshape(cfg.numberOfHeads, cfg.headSize, -1)
        rows[heads] = rows[heads].astype(np.float32) * np.float32(query)
        d, _ = _blocks(tensors, TensorRole.ATTENTION_KEY, cfg.dim)
        d[:] = d.astype(np.float32) * np.float32(key)
    return edit


@pytest.mark.parametrize("heads,kv_heads,head", [(4, 4, 64), (8, 4, 64), (8, 2, 64), (8, 1, 64), (2, 2, 128), (4, 2, 128), (8, 2, 128), (8, 1, 128)])
def test_range_and_tile_edges(dev, heads, kv_heads, head):
    errors = attention_errors(dev, _rope, heads, kv_heads, head, 16, [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 192])
    assert max(errors) < BAR, errors


@pytest.mark.parametrize("page,depths,width", [(16, [1279, 1280, 1281, 2600], 1), (1, [700, 1281], 1), (16, [300, 900], 3)])
def test_many_ranges_pages_and_rows(dev, page, depths, width):
    errors = attention_errors(dev, _rope, 8, 2, 64, page, depths, width)
    assert max(errors) < BAR, errors


@pytest.mark.parametrize("heads,kv_heads,head,depths", [
    (8, 2, 64, [255, 256, 257, 767, 768, 769, 1791, 1792, 1793, 2303, 2304, 2305, 2367, 2368, 2369]), (8, 8, 64, [1279, 1280, 1281, 2560, 2561]),
    (8, 1, 128, [256, 257, 768, 769, 2304, 2305, 2368, 2369])])
def test_folds_of_many_ranges(dev, heads, kv_heads, head, depths):
    errors = attention_errors(dev, _rope, heads, kv_heads, head, 16, depths)
    assert max(errors) < BAR, errors


@pytest.mark.parametrize("heads,kv_heads,head", [(4, 4, 64), (8, 2, 64), (8, 1, 64), (8, 2, 128), (8, 1, 128)])
@pytest.mark.parametrize("query,key", [(2.0 ** -6, 2.0 ** 6), (2.0 ** -12, 2.0 ** 12), (2.0 ** 15, 2.0 ** -13)])
def test_queries_of_every_magnitude(dev, heads, kv_heads, head, query, key):
    """Small queries against large keys, and queries beyond binary16 against small ones: scores of the same size as ever (four times
    it in the last case), so the same bar: a query keeps its bits whatever its magnitude."""
    outs = attention_outputs(dev, _rope, heads, kv_heads, head, 16, [3, 70, 300], edit=_scaled(query, key))
    most = max(float(np.abs(q).max()) for _, _, q in outs)
    assert most > 65504 if query > 1 else most < 8 * query, most
    errors = [rel_l2(got.reshape(-1), want.reshape(-1)) for got, want, _ in outs]
    assert max(errors) < BAR, errors


@pytest.mark.parametrize("heads,kv_heads,head", [(8, 4, 64), (8, 2, 64), (8, 1, 64), (8, 2, 128), (8, 1, 128)])
def test_large_head_beside_ordinary_ones(dev, heads, kv_heads, head):
    """The heads that share a KV head with one whose query is 2^25 times as large lose nothing by it."""
    group = heads // kv_heads
    for got, want, q in attention_outputs(dev, _rope, heads, kv_heads, head, 16, [3, 70, 300], edit=_scaled(2.0 ** 25, 1.0, slice(0, None, group))):
        assert np.abs(q[::group]).max() > 65504 and np.isfinite(got).all()
        errors = [rel_l2(got[h], want[h]) for h in range(heads) if h % group != 0]
        assert max(errors) < BAR, errors


KEY, VALUE = 1, 2  # tokens whose key (value) goes beyond binary16 in some components: infinite in the pages


def _overflow(cfg, tensors):
    """Embedding columns 0 and 32 are zero for all tokens but KEY and VALUE; key component 0 and value component 5 of every KV head
    weigh these columns with more than 6e4."""
    d, q = _blocks(tensors, TensorRole.TOKEN_EMBEDDING, cfg.dim, -1)
    q[:, 0:2, 0] = 0
    for block, token in ((0, KEY), (1, VALUE)):
        d[token, block], q[token, block] = 1.0, 0
        q[token, block, 0] = 127
    for role, block, component in ((TensorRole.ATTENTION_KEY, 0, 0), (TensorRole.ATTENTION_VALUE, 1, 5)):
        d, q = _blocks(tensors, role, cfg.dim)
        rows = slice(component, None, cfg.headSize)
        d[rows, block], q[rows, block] = 500.0, 0
        q[rows, block, 0] = 127


@pytest.mark.parametrize("heads,kv_heads,head", [(8, 8, 64), (8, 4, 64), (8, 2, 64), (8, 1, 64), (8, 4, 128), (8, 2, 128), (8, 1, 128)])
@pytest.mark.parametrize("pos,special,token", [
    (70, {0: KEY}, 5),        # scores of +inf (the output is NaN) or -inf (no weight) by the sign of the query
    (300, {101: KEY}, 5),     # the same, or NaN, in one of five ranges
    (66, {32: KEY}, 5),       # the same, the only key of a warp's sixteen
    (16, {}, KEY),            # the same, the step's own key
    (300, {101: VALUE}, 5),   # an output of +-inf
    (16, {}, VALUE),
    (130, {3: KEY, 127: VALUE}, 5)])
def test_infinite_keys_and_values(dev, heads, kv_heads, head, pos, special, token):
    outs = []
    for seed in (3, 4, 5):
        outs += attention_outputs(dev, _rope, heads, kv_heads, head, 16, [pos], seed=seed, edit=_overflow, special=special, token=token)
    keys = KEY in special.values() or token == KEY
    values = VALUE in special.values() or token == VALUE
    nan = np.concatenate([np.isnan(want).all(axis=1) for _, want, _ in outs])
    assert not keys or (nan.any() and not nan.all())
    assert not values or any(np.isinf(want[:, 5]).any() for _, want, _ in outs)
    for got, want, _ in outs:
        assert np.array_equal(np.isnan(got), np.isnan(want))
        inf = np.isinf(want)
        assert np.array_equal(got[inf], want[inf])
        for h in range(heads):
            fine = np.isfinite(want[h])
            assert not fine.any() or rel_l2(got[h][fine], want[h][fine]) < BAR


def test_nan_key(dev):
    """Positions that nothing was written to hold NaN: an output that attends to one is NaN."""
    cfg = jl.Configuration(dim=512, hiddenDim=512, numberOfLayers=1, numberOfHeads=8, numberOfKeyValueHeads=2, vocabularySize=512, contextLength=128)
    model = jl.load_model(dev, cfg, jl.synth_model_tensors(cfg, GGMLType.Q8_0, seed=3, std=0.05), *_rope(cfg))
    kv = model.createKvStorage(jl.KvStorageRequest(8, 8, 1, 16, 1, cfg.kvDim))
    kv.publishBlockTable(np.arange(8, dtype=np.int32))
    kv.fill(0x7E00)
    boundary = jl.B200InvocationBoundary(model, kvSlot=0)
    boundary.prefill(np.arange(32, dtype=np.int32), 0)
    boundary.prefill(np.arange(33, 65, dtype=np.int32), 33)
    jl.B200BatchExecutor(model).decodeStep(jl.BatchSlots([True], [5], [65], [0]))
    assert np.isnan(model.debugRead("xb")).all()
    kv.close()
