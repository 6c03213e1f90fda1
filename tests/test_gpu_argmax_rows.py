"""The greedy token of every row of a wide decode launch is the first index of that row's maximum: exact, over
vocabularies whose rows start on 16 bytes and ones whose rows do not, around one sweep of a CTA (32 768 logits in
16-byte loads, 8192 in 4-byte loads), with exact ties planted before and after the maximum."""
import numpy as np
import pytest

import jitllm_b200 as jl
from jitllm_b200 import GGMLType

from tests.util import small_config

pytestmark = pytest.mark.gpu

WIDTH = 16


def _decode(dev, cfg, tensors, tokens):
    cr, ci = jl.precomputeFreqsCis(cfg.contextLength, cfg.headSize, cfg.ropeTheta)
    model = jl.load_model(dev, cfg, tensors, cr, ci, maxBatch=WIDTH)
    kv = model.createKvStorage(jl.KvStorageRequest(2 * WIDTH, 2, WIDTH, 16, cfg.numberOfLayers, cfg.kvDim))
    kv.publishBlockTable(np.arange(2 * WIDTH, dtype=np.int32))
    out, logits = jl.B200BatchExecutor(model).decodeStep(
        jl.BatchSlots([True] * WIDTH, tokens, [0] * WIDTH, list(range(WIDTH))), wantLogits=True)
    kv.close()
    return [int(v) for v in out], np.array(logits)


@pytest.mark.parametrize("vocab", [37, 1000, 4097, 8193, 32768, 32772, 40002])
def test_first_index_of_the_maximum(dev, vocab):
    cfg = small_config(layers=1, ctx=32, vocab=vocab)
    tensors = jl.synth_model_tensors(cfg, GGMLType.Q8_0, seed=vocab, std=0.05)
    tokens = [int(v) for v in np.random.default_rng(vocab).integers(0, vocab, size=WIDTH)]
    out, logits = _decode(dev, cfg, tensors, tokens)
    assert out == [int(v) for v in np.argmax(logits, axis=1)]

    # row 0's best token gets copies at other indexes: the weights are equal, so the logits tie exactly
    t, w = tensors[(jl.TensorRole.OUTPUT, -1)]
    w = w.copy()
    rb = cfg.dim // 32 * 34
    best = out[0]
    copies = sorted({0, best, (best + 1) % vocab, (best + vocab // 2) % vocab, vocab - 1})
    for j in copies:
        w[j * rb:(j + 1) * rb] = tensors[(jl.TensorRole.OUTPUT, -1)][1][best * rb:(best + 1) * rb]
    tensors[(jl.TensorRole.OUTPUT, -1)] = (t, w)
    out, logits = _decode(dev, cfg, tensors, tokens)
    assert len({float(logits[0][j]) for j in copies}) == 1
    assert out == [int(v) for v in np.argmax(logits, axis=1)]
    assert out[0] == copies[0] == 0
