"""The tensor-core (tcgen05) matrix-matrix path against the oracle's batch matmul
(FloatTensor.matmul(context, that[], out[], ...)): per-matmul relative L2 <= 1e-3 is the stated
bar. Weights are rounded to fp16 after an element-exact fp32 decode and activations are carried
as fp16 hi+lo, so ~3e-4 is expected."""
import numpy as np
import pytest

import jitllm_b200 as jl
from jitllm_b200 import GGMLType
from tests.util import rel_l2

pytestmark = pytest.mark.gpu
BAR = 1e-3
EXPECT = 6e-4
FORMATS = [GGMLType.Q8_0, GGMLType.Q4_0, GGMLType.Q4_K]


@pytest.mark.parametrize("t", FORMATS)
@pytest.mark.parametrize("rows,cols,n", [(128, 256, 8), (256, 512, 16), (200, 768, 9), (384, 1024, 33),
                                         (1000, 2048, 64), (130, 256, 130), (512, 1792, 200)])
def test_small_and_ragged_tiles(dev, oracle, t, rows, cols, n):
    w = jl.synth_tensor(t, rows * cols, seed=rows + cols + n)
    x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
    got, want = dev.matmul(t, w, rows, cols, x), oracle.matmul(t, w, x, rows, cols)
    assert got.shape == (n, rows)
    err = rel_l2(got, want)
    assert err < BAR and err < EXPECT, err
    # every row individually, so a misplaced tile cannot hide in the aggregate
    per_row = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert per_row.max() < BAR, per_row.max()


@pytest.mark.parametrize("t", FORMATS)
@pytest.mark.parametrize("rows,cols,n", [(4096, 4096, 32), (14336, 4096, 8), (4096, 14336, 32)])
def test_sweep_shapes(dev, oracle, t, rows, cols, n):
    w = jl.synth_tensor(t, rows * cols, seed=rows + n + int(t))
    x = np.random.default_rng(3).standard_normal((n, cols)).astype(np.float32)
    got, want = dev.matmul(t, w, rows, cols, x), oracle.matmul(t, w, x, rows, cols)
    err = rel_l2(got, want)
    assert err < BAR and err < EXPECT, err


def test_prefill_sized_batch_q8_0(dev, oracle):
    rows, cols, n, t = 4096, 4096, 512, GGMLType.Q8_0
    w = jl.synth_tensor(t, rows * cols, seed=17)
    x = np.random.default_rng(5).standard_normal((n, cols)).astype(np.float32)
    got = dev.matmul(t, w, rows, cols, x)
    sample = [0, 1, 127, 128, 255, 300, 511]
    want = oracle.matmul(t, w, x[sample], rows, cols)
    assert rel_l2(got[sample], want) < EXPECT
    # linearity at full size: W(a + b) = W a + W b up to the operand rounding
    y2 = dev.matmul(t, w, rows, cols, x[:64] + x[64:128])
    assert rel_l2(y2, got[:64] + got[64:128]) < BAR


def test_wide_activations_do_not_overflow_fp16(dev, oracle):
    rows, cols, n, t = 256, 1024, 16, GGMLType.Q4_K
    w = jl.synth_tensor(t, rows * cols, seed=19)
    x = (np.random.default_rng(6).standard_normal((n, cols)) * 300.0).astype(np.float32)
    got, want = dev.matmul(t, w, rows, cols, x), oracle.matmul(t, w, x, rows, cols)
    assert rel_l2(got, want) < EXPECT


def test_tall_product(dev, oracle):
    """The most weight rows against more than a thousand activation rows: 501 row tiles by six token tiles in one launch, an
    arrival counter for either CTA of each. (Without the workspace of the split activations the same product goes in token
    slabs: test_wide_product_inside_a_capture.)"""
    rows, cols, n, t = 128256, 256, 1100, GGMLType.Q4_0
    w = jl.synth_tensor(t, rows * cols, seed=23)
    x = np.random.default_rng(7).standard_normal((n, cols)).astype(np.float32)
    got = dev.matmul(t, w, rows, cols, x)
    assert got.shape == (n, rows)
    sample = [0, 63, 64, 1023, 1024, 1025, 1099]
    want = oracle.matmul(t, w, x[sample], rows, cols)
    assert rel_l2(got[sample], want) < EXPECT


@pytest.mark.parametrize("t", FORMATS)
def test_widest_sweep_batch(dev, oracle, t):
    """N = 2048, the widest batch of the standalone sweep, on the 14336 x 4096 shape: sampled token
    rows against the oracle (the full product is 120 G multiply-adds on the CPU), rows on either side
    of token-tile boundaries among them."""
    rows, cols, n = 14336, 4096, 2048
    w = jl.synth_tensor(t, rows * cols, seed=29 + int(t))
    x = np.random.default_rng(8).standard_normal((n, cols)).astype(np.float32)
    got = dev.matmul(t, w, rows, cols, x)
    assert got.shape == (n, rows)
    sample = [0, 127, 128, 1023, 1024, 1900, 2047]
    want = oracle.matmul(t, w, x[sample], rows, cols)
    err = rel_l2(got[sample], want)
    assert err < BAR and err < EXPECT, err
    assert np.all(np.isfinite(got))


@pytest.mark.parametrize("t", FORMATS + [GGMLType.Q4_1, GGMLType.Q5_K, GGMLType.Q6_K])
@pytest.mark.parametrize("rows,cols,n", [(100, 256, 129),     # one tile, half of it (and most of the token half) empty
                                         (256, 512, 256),     # exactly one tile of 256 tokens
                                         (300, 2048, 257),    # a second row tile and a second token tile of one row
                                         (1536, 4096, 470),   # 18 tiles on 74 CTA pairs: several pairs per tile
                                         (6144, 1024, 513),   # 72 tiles on 72 pairs: ranges aligned to tiles
                                         (12900, 512, 300)])  # 102 tiles: ranges end inside tiles
def test_wide_products_on_cta_pairs(dev, oracle, t, rows, cols, n):
    """More than 128 rows: tiles of 256 weight rows on CTA pairs. Same operands as the narrow kernel (weights rounded once to
    binary16, 2^-12 relative on average; activations in 22 bits), so the same expected error."""
    make = jl.synth_tensor if t in FORMATS else jl.random_blocks
    w = make(t, rows * cols, seed=rows + cols + n)
    x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
    got = dev.matmul(t, w, rows, cols, x)
    sample = sorted({0, 1, 127, 128, 255, 256, n // 2, n - 2, n - 1} & set(range(n)))
    want = oracle.matmul(int(t), w, x[sample], rows, cols)
    err = np.linalg.norm(got[sample] - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < EXPECT, err
    assert np.all(np.isfinite(got))
    assert np.array_equal(dev.matmul(t, w, rows, cols, x), got)  # partial tiles are added in a fixed order


@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q8_0])
@pytest.mark.parametrize("n", [191, 192,        # one tile of 192 tokens
                               193, 255, 256,   # one tile of 256, in two passes
                               257, 384, 385,   # tiles of 192 again
                               576, 577])
def test_wide_products_over_the_tile_widths(dev, oracle, t, n):
    """Rows on either side of every token-tile edge and of the CTAs' halves of the tiles, in both forms of the CTA-pair
    kernel; 300 weight rows (a half-empty row tile) and 2048 columns (32 operand stages: several rounds of every ring)."""
    rows, cols = 300, 2048
    w = jl.synth_tensor(t, rows * cols, seed=n)
    x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
    got = dev.matmul(t, w, rows, cols, x)
    half = 128 if 192 < n <= 256 else 96
    edges = [e for k in range(half, n, half) for e in (k - 1, k)]
    sample = sorted({0, n - 1, *edges} & set(range(n)))
    want = oracle.matmul(t, w, x[sample], rows, cols)
    err = np.linalg.norm(got[sample] - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < EXPECT, err
    assert np.all(np.isfinite(got))
    assert np.array_equal(dev.matmul(t, w, rows, cols, x), got)


def test_wide_product_is_as_close_to_64_bits_as_the_narrow_one(dev):
    """The same rows through the 128-row kernel (an accumulator for either part of the activations) and, as part of a
    wider block, through the CTA pairs. The weights are whole multiples of 2^-7, exact in binary16, so what is left is the
    activations' 22 bits and the binary32 sums: 256 steps over 4096 columns that are cut off at the accumulator's last
    place, 256 * 2^-24 = 1.5e-5 at most. 148 row tiles of 128 and 74 of 256: every sum runs over whole rows, also in the form that walks a tile twice (256 rows)
    and in the one with two accumulators (384)."""
    rows, cols, n = 148 * 128, 4096, 384
    rng = np.random.default_rng(3)
    q = rng.integers(-127, 128, size=(rows, cols)).astype(np.int8)
    blocks = np.empty((rows, cols // 32, 34), np.uint8)
    blocks[:, :, :2] = np.frombuffer(np.float16(2.0 ** -7).tobytes(), np.uint8)
    blocks[:, :, 2:] = q.reshape(rows, cols // 32, 32).view(np.uint8)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    pick = np.sort(rng.choice(rows, 256, replace=False))
    want = x.astype(np.float64) @ (q[pick].astype(np.float64) * 2.0 ** -7).T
    err = {}
    for m in (128, 256, n):
        got = dev.matmul(GGMLType.Q8_0, blocks.reshape(-1), rows, cols, x[:m])[:, pick]
        err[m] = np.linalg.norm(got[:128] - want[:128]) / np.linalg.norm(want[:128])
    assert max(err.values()) < 256 * 2.0 ** -24, err
    assert max(err.values()) <= 1.05 * err[128], err


@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q8_0])
@pytest.mark.parametrize("tail", [9, 33, 100, 300])  # a second slab for the 16-, 64- and 128-row kernels and the CTA pairs
def test_wide_product_in_two_slabs(dev, oracle, t, tail):
    """14336 columns: 1152 rows of split activations fill the workspace, the rest go in a second slab with a descriptor of
    its own, behind the first slab's product on the same buffer."""
    rows, cols, n = 300, 14336, 1152 + tail
    w = jl.synth_tensor(t, rows * cols, seed=tail)
    x = np.random.default_rng(tail).standard_normal((n, cols)).astype(np.float32)
    got = dev.matmul(t, w, rows, cols, x)
    sample = [0, 191, 192, 1150, 1151, 1152, 1153, n - 2, n - 1]
    want = oracle.matmul(t, w, x[sample], rows, cols)
    err = np.linalg.norm(got[sample] - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < EXPECT, err
    assert np.all(np.isfinite(got))


def test_split_workspace_is_there_from_the_first_wide_product_on(built):
    """A context that never multiplies a stand-alone matrix by more than 64 rows does not hold the 64 MiB their activations
    are split into; the first that does takes it, later ones find it, and it goes with the context."""
    import torch
    t, rows, cols = GGMLType.Q8_0, 256, 512
    w = jl.synth_tensor(t, rows * cols, seed=3)
    x = np.random.default_rng(3).standard_normal((70, cols)).astype(np.float32)
    free = lambda: torch.cuda.mem_get_info(0)[0] / 2 ** 20
    with jl.Device(0) as warm:  # the kernels' code is loaded once per process
        want = warm.matmul(t, w, rows, cols, x)
        warm.matmul(t, w, rows, cols, x[:64])
        before = free()
        with jl.Device(0) as d:
            narrow = d.matmul(t, w, rows, cols, x[:64])
            held = before - free()
            assert held < 64 + 32, held  # the products' own scratch is 64 MiB
            assert np.array_equal(d.matmul(t, w, rows, cols, x), want)
            assert 60 <= before - free() - held <= 70
            assert np.array_equal(d.matmul(t, w, rows, cols, x), want)
            assert 60 <= before - free() - held <= 70
        assert abs(before - free()) < 8
    assert np.linalg.norm(narrow - want[:64]) < EXPECT * np.linalg.norm(want[:64])


@pytest.mark.parametrize("rows,cols,n", [(300, 512, 100),        # two token tiles of the in-kernel conversion
                                         (128256, 256, 1100)])   # and more tiles than arrival counters: two token slabs
def test_wide_product_inside_a_capture(built, oracle, rows, cols, n):
    """The first wide product of a context while its stream is being captured, where no memory can be taken: the activations
    are converted inside the product kernel, the capture stays whole, and its replay gives the product."""
    import torch
    t = GGMLType.Q4_0
    w = jl.synth_tensor(t, rows * cols, seed=23)
    x = np.random.default_rng(7).standard_normal((n, cols)).astype(np.float32)
    with jl.Device(0) as d:
        m = d.upload_matrix(t, w, rows, cols)
        xd, yd = d.alloc(x.nbytes), d.alloc(n * rows * 4)
        d.h2d(xd, x)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(d._lib.jl_stream(d.handle))):
            m.matmul_dev(xd, n, yd)
        graph.replay()
        torch.cuda.synchronize()
        got = np.empty((n, rows), np.float32)
        d.d2h(got, yd)
        del graph
        m.close()
    sample = sorted({0, 63, 64, 65, n // 2, n - 1} | ({1023, 1024, 1025} & set(range(n))))
    want = oracle.matmul(t, w, x[sample], rows, cols)
    err = np.linalg.norm(got[sample] - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < EXPECT, err
