"""Decode attention of wide launches (one CTA per row and KV head, sixteen keys to a warp at a time) at the depths where a
warp's group, a round of the four warps or the ring of three groups begins and ends: against the oracle's logits, and bit
for bit across page sizes, since the page size chooses how a group is addressed and nothing else."""
import numpy as np
import pytest

import jitllm_b200 as jl
from jitllm_b200 import GGMLType

pytestmark = pytest.mark.gpu

WIDTH = 64
DEPTHS = [0, 1, 15, 16, 17, 31, 32, 47, 48, 63, 64, 65, 79, 80, 127, 128, 129, 143, 144, 191, 192, 193, 207, 208, 209, 255, 256, 257]


def _logits(dev, cfg, tensors, rope, page, prompt):
    model = jl.load_model(dev, cfg, tensors, *rope, maxBatch=WIDTH)
    bps = (cfg.contextLength + page - 1) // page
    kv = model.createKvStorage(jl.KvStorageRequest(WIDTH * bps, bps, WIDTH, page, cfg.numberOfLayers, cfg.kvDim))
    kv.publishBlockTable(np.random.default_rng(page).permutation(WIDTH * bps).astype(np.int32))
    kv.fill(0x7E00)  # NaN wherever nothing was written
    rows = [DEPTHS[b % len(DEPTHS)] for b in range(WIDTH)]
    for b, n in enumerate(rows):
        if n > 0:
            jl.B200InvocationBoundary(model, kvSlot=b).prefill(prompt[:n], 0)
    active = [b != 7 for b in range(WIDTH)]
    _, logits = jl.B200BatchExecutor(model).decodeStep(
        jl.BatchSlots(active, [5] * WIDTH, rows, list(range(WIDTH))), wantLogits=True)
    kv.close()
    return rows, active, np.array(logits)


@pytest.mark.parametrize("heads,kv_heads,head", [(4, 4, 64), (8, 4, 64), (16, 4, 64), (16, 2, 64), (4, 2, 128), (8, 2, 128)])
def test_group_edges_and_page_sizes(dev, oracle, heads, kv_heads, head):
    cfg = jl.Configuration(dim=heads * head, hiddenDim=512, numberOfLayers=1, numberOfHeads=heads, numberOfKeyValueHeads=kv_heads,
                           vocabularySize=512, contextLength=max(DEPTHS) + 16)
    tensors = jl.synth_model_tensors(cfg, GGMLType.Q8_0, seed=heads + head, std=0.05)
    om = oracle.Model(cfg, tensors)
    prompt = np.random.default_rng(heads).integers(0, cfg.vocabularySize, size=max(DEPTHS)).astype(np.int32)
    rope = om.rope_tables()
    rows, active, logits = _logits(dev, cfg, tensors, rope, 16, prompt)
    for i, t in enumerate(prompt):
        om.forward(int(t), i)
    want = {pos: np.array(om.forward(5, pos)) for pos in sorted(DEPTHS, reverse=True)}  # overwrites its own key: deepest first
    for b in range(WIDTH):
        if active[b]:
            assert float(np.max(np.abs(logits[b] - want[rows[b]]))) < 1e-2, (b, rows[b])
    for page in (1, 12, 24, 48):
        _, _, other = _logits(dev, cfg, tensors, rope, page, prompt)
        assert np.array_equal(logits[active], other[active]), page
