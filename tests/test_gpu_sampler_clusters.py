"""Sampling at the widths where the number of CTAs that share a row changes (8 up to 16 rows, 4 up to 32, 2 beyond): the tokens
of the oracle's restatement of the reference's chain, exactly, at vocabularies whose slices are ragged. (At a few thousand
tokens the reference's fp32 sums are off by at most some 1e-6 of the mass, so only a draw that near to a boundary of the
distribution may go to the neighbour.) Vocabularies of real size, where a thread of four or two CTAs has more elements than it
keeps in registers: the token whose interval of the 64-bit cumulative distribution holds the draw."""
import numpy as np
import pytest

from tests.test_gpu_sampler import _model, _step_and_sample, _within_float64_interval

pytestmark = pytest.mark.gpu
# Of the mass: the device's exponentials are within 2 units of the last place (2.4e-7), its sums cut each off at 2^-40 (1.2e-7 for
# 128 256 of them, the largest being 1), the nucleus' mass and the draw times it are rounded to binary32 (6e-8 each): under 6e-7.
EPS = 1e-6


@pytest.mark.parametrize("vocab", [131, 5003])
@pytest.mark.parametrize("width", [16, 17, 32, 33, 64])
def test_tokens_at_every_cluster_width(dev, oracle, width, vocab):
    cfg, model, kv = _model(dev, vocab, width, std=0.3)
    rng = np.random.default_rng(width * vocab)
    active = [b % 9 != 4 for b in range(width)]
    for temperature, topp in ((0.8, 0.95), (1.3, 0.5), (1.0, 0.0)):
        tokens = [int(v) for v in rng.integers(0, vocab, size=width)]
        u = [np.float32(int(rng.random() * (1 << 24)) / (1 << 24)) for _ in range(width)]
        logits, got = _step_and_sample(dev, model, width, tokens, temperature, topp, u, active=active)
        for b in range(width):
            if not active[b]:
                assert got[b] == -1
                continue
            want, margin = oracle.sample(logits[b], temperature, topp, float(u[b]))
            assert int(got[b]) == want or margin < 2e-6, (b, int(got[b]), want, margin)
    kv.close()


@pytest.mark.parametrize("vocab", [70001, 128256])
@pytest.mark.parametrize("width", [17, 33, 64])
def test_more_elements_than_a_thread_keeps(dev, width, vocab):
    cfg, model, kv = _model(dev, vocab, width, std=0.3)
    rng = np.random.default_rng(width + vocab)
    for temperature, topp in ((0.8, 0.95), (1.5, 0.5), (1.0, 0.0)):
        tokens = [int(v) for v in rng.integers(0, vocab, size=width)]
        u = [np.float32(int(rng.random() * (1 << 24)) / (1 << 24)) for _ in range(width)]
        logits, got = _step_and_sample(dev, model, width, tokens, temperature, topp, u)
        for b in range(width):
            assert _within_float64_interval(logits[b], temperature, topp, float(u[b]), int(got[b]), eps=EPS), (b, int(got[b]))
    kv.close()
