"""Decode attention with the keys split over CTAs, by itself: the attention output of a one-layer model's step against a 64-bit
softmax over the query, keys and values that the device itself used (the projections and pages are read back), at the depths
where the split changes: one key, around one tile of 64, where a second range, a third and the last of twenty begin, and
where ranges grow beyond a tile; every head size and group."""
import numpy as np
import pytest

import jitllm_b200 as jl
from jitllm_b200 import GGMLType
from tests.util import rel_l2

pytestmark = pytest.mark.gpu
# A score is a sum of head_dim exact products, added sixteen at a time into binary32: at most 8 + 3 additions cut off or rounded
# at 2^-23 of a partial sum of some 10, so 1e-5 of a weight in the worst case; outputs average the weights' errors.
BAR = 1e-5


def attention_errors(dev, rope, heads, kv_heads, head, page, depths, width=1, std=0.05, seed=3):
    """rel-L2 of the attention outputs of one step at every depth (keys in the pages before it)."""
    cfg = jl.Configuration(dim=heads * head, hiddenDim=512, numberOfLayers=1, numberOfHeads=heads, numberOfKeyValueHeads=kv_heads,
                           vocabularySize=512, contextLength=max(depths) + 16)
    tensors = jl.synth_model_tensors(cfg, GGMLType.Q8_0, seed=seed, std=std)
    cr, ci = rope(cfg)
    model = jl.load_model(dev, cfg, tensors, cr, ci, maxBatch=width)
    bps = (cfg.contextLength + page - 1) // page
    kv = model.createKvStorage(jl.KvStorageRequest(width * bps, bps, width, page, 1, cfg.kvDim))
    kv.publishBlockTable(np.random.default_rng(seed).permutation(width * bps).astype(np.int32))
    kv.fill(0x7E00)  # NaN wherever nothing was written
    rng = np.random.default_rng(seed + 1)
    prompt = rng.integers(0, cfg.vocabularySize, size=max(depths)).astype(np.int32)
    for b in range(width):
        jl.B200InvocationBoundary(model, kvSlot=b).prefill(prompt if max(depths) > 0 else [1], 0)
    ex = jl.B200BatchExecutor(model)
    cr, ci = np.asarray(cr, dtype=np.float32).reshape(-1, head // 2), np.asarray(ci, dtype=np.float32).reshape(-1, head // 2)
    out = []
    for pos in sorted(depths, reverse=True):  # the step overwrites the key at its position: deepest first
        rows = [max(0, pos - 3 * b) for b in range(width)]
        ex.decodeStep(jl.BatchSlots([True] * width, [5 + b for b in range(width)], rows, list(range(width))))
        for b, p in enumerate(rows):
            q = model.debugRead("q", b).reshape(heads, head // 2, 2)
            q = np.stack([q[..., 0] * cr[p] - q[..., 1] * ci[p], q[..., 0] * ci[p] + q[..., 1] * cr[p]], axis=-1)
            q = q.reshape(heads, head).astype(np.float64)
            k, v = (np.stack([kv.readRow(w, b, 0, i).view(np.float16) for i in range(p + 1)]).astype(np.float64).reshape(p + 1, kv_heads, head)
                    for w in ("k", "v"))
            got = model.debugRead("xb", b)
            want = np.empty((heads, head))
            for h in range(heads):
                s = k[:, h * kv_heads // heads] @ q[h] / np.sqrt(head)
                w = np.exp(s - s.max())
                want[h] = (w / w.sum()) @ v[:, h * kv_heads // heads]
            out.append(rel_l2(got, want.reshape(-1)))
    kv.close()
    return out


def _rope(cfg):
    return jl.precomputeFreqsCis(cfg.contextLength, cfg.headSize, cfg.ropeTheta)


@pytest.mark.parametrize("heads,kv_heads,head", [(4, 4, 64), (8, 4, 64), (8, 2, 64), (8, 1, 64), (2, 2, 128), (4, 2, 128), (8, 2, 128), (8, 1, 128)])
def test_range_and_tile_edges(dev, heads, kv_heads, head):
    errors = attention_errors(dev, _rope, heads, kv_heads, head, 16, [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 192])
    assert max(errors) < BAR, errors


@pytest.mark.parametrize("page,depths,width", [(16, [1279, 1280, 1281, 2600], 1), (1, [700, 1281], 1), (16, [300, 900], 3)])
def test_many_ranges_pages_and_rows(dev, page, depths, width):
    errors = attention_errors(dev, _rope, 8, 2, 64, page, depths, width)
    assert max(errors) < BAR, errors


def test_queries_beyond_binary16(dev):
    """Query weights of a size that takes the rotated query past 65504: the kernel scales it before it is split."""
    errors = attention_errors(dev, _rope, 4, 1, 64, 16, [3, 70], std=40.0)
    assert all(np.isfinite(errors)) and max(errors) < 1e-3, errors  # scores of 1e5 and more: their last bits decide
