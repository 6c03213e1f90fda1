"""The counters of bytes that go up and come down count what is copied: a step's inputs go up in one copy of sixteen bytes per row
(token, position, slot, and the active flag in a word of its own)."""
import numpy as np
import pytest

import jitllm_b200 as jl
from jitllm_b200 import GGMLType

from tests.util import small_config

pytestmark = pytest.mark.gpu


def test_bytes_of_steps_prompts_and_generation(dev):
    cfg = small_config(layers=1)
    cr, ci = jl.precomputeFreqsCis(cfg.contextLength, cfg.headSize, cfg.ropeTheta)
    model = jl.load_model(dev, cfg, jl.synth_model_tensors(cfg, GGMLType.Q8_0, seed=2), cr, ci, maxBatch=5)
    kv = model.createKvStorage(jl.KvStorageRequest(20, 4, 5, 16, cfg.numberOfLayers, cfg.kvDim))
    kv.publishBlockTable(np.arange(20, dtype=np.int32))
    ex = jl.B200BatchExecutor(model)

    def moved(call):
        before = dev.counters()
        call()
        after = dev.counters()
        return tuple(after[k] - before[k] for k in ("h2d_bytes", "d2h_bytes"))

    batch = jl.BatchSlots([True, False, True, True, True], [1, 2, 3, 4, 5], [0] * 5, list(range(5)))
    assert moved(lambda: ex.decodeStep(batch)) == (16 * 5, 4 * 5 + 4)
    assert moved(lambda: ex.decodeStep(batch, sampler=jl.Sampler.selectSampler(cfg.vocabularySize, 0.8, 0.9, 1))) == (20 * 5, 8 * 5 + 4)
    assert moved(lambda: ex.generate(batch, 3)) == (16 * 5, 4 * 15 + 4)
    assert moved(lambda: jl.B200InvocationBoundary(model, kvSlot=1).prefill(np.arange(9, dtype=np.int32), 0))[0] == 16 * 9
    assert moved(lambda: jl.B200InvocationBoundary(model, kvSlot=1).prefill(np.arange(2, dtype=np.int32), 9))[0] == 16 * 2
    kv.close()
