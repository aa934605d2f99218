"""The batch kernel (gemv_batch.cu) against the CPU oracle on a B200, through the public wrapper, at the edges of its tiles and
operands.  The size rule of `ggq_gemv` would hand small shapes to other kernels; it is off here (the switch is read once per process, so the
tests run in a child process).

Bars: float32 output within 2e-5 relative L2 of the oracle's double-accumulated product, as for the other exact kernels (float32 summation
order is all that separates them); a one-hot activation returns the decoded weight times the activation exactly; a launch repeats bit for
bit; outputs that are not finite are what the decoded weights give."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

from gguf_jax_b200 import QuantizedArray, kernels, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FORMATS = [QT.Q2_K, QT.Q3_K, QT.Q4_K, QT.Q5_K, QT.Q6_K, QT.IQ4_XS, QT.IQ2_XXS, QT.IQ2_XS, QT.IQ2_S, QT.IQ3_XXS, QT.IQ3_S, QT.IQ1_S, QT.IQ1_M,
           QT.TQ1_0, QT.TQ2_0]
ALWAYS = os.environ.get("GGQ_TILE_ALWAYS") == "1"


@pytest.mark.skipif(ALWAYS, reason="the child process")
def test_with_the_size_rule_off():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.abspath(__file__), "-q", "-x", "-m", "gpu"],
                       env=dict(os.environ, GGQ_TILE_ALWAYS="1"), cwd=root, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:] + r.stderr[-1000:]


def product(xb, wb, qt, n, k, dtype=torch.float32):
    w = QuantizedArray.from_bytes(wb, qt, shape=(n, k), device="cuda")
    return kernels.fused_matmul(torch.from_numpy(xb).cuda().to(torch.bfloat16), w, out_dtype=dtype).cpu()


@pytest.mark.skipif(not ALWAYS, reason="runs in the child process")
@pytest.mark.parametrize("qtype", FORMATS, ids=lambda t: t.name)
def test_edges_of_tiles_and_splits(qtype):
    # one row and one block; a ragged last tile; rows that are not 16-byte aligned (odd numbers of blocks); one and two column tiles, full
    # and ragged; clusters and, at K = 29 * 1024, passes
    for n, k in [(1, 256), (17, 768), (40, 2048), (2500, 1280), (33, 29 * 1024)]:
        wb = synth.make_weight_bytes(n, k, qtype, seed=n)
        for m in (5, 8, 9, 16):
            xb = synth.make_x(m, k, seed=m)
            got = product(xb, wb, qtype, n, k).numpy()
            assert O.rel_l2(got, O.c_matmul(O.bf16_bits(xb), wb, qtype)) <= 2e-5, (n, k, m)
            assert np.array_equal(got.view(np.uint32), product(xb, wb, qtype, n, k).numpy().view(np.uint32))
            assert torch.equal(product(xb, wb, qtype, n, k, torch.bfloat16), torch.from_numpy(got).to(torch.bfloat16))


@pytest.mark.skipif(not ALWAYS, reason="runs in the child process")
@pytest.mark.parametrize("qtype", FORMATS, ids=lambda t: t.name)
def test_one_hot_returns_the_weight(qtype):
    n, k, m = 32, 512, 16
    wb = synth.make_weight_bytes(n, k, qtype, seed=3)
    dense = O.c_dequantize(wb, qtype).reshape(n, k).astype(np.float32)
    for first in range(0, k, m):
        xb = np.zeros((m, k), np.float32)
        xb[np.arange(m), first + np.arange(m)] = 2.0 ** (np.arange(m) * 9 - 70)
        got = product(xb, wb, qtype, n, k).numpy()
        assert np.array_equal(got, (dense[:, first:first + m] * xb[np.arange(m), first + np.arange(m)]).T)


@pytest.mark.skipif(not ALWAYS, reason="runs in the child process")
@pytest.mark.parametrize("qtype", FORMATS, ids=lambda t: t.name)
def test_magnitudes_over_the_whole_range(qtype):
    # a block whose activations span 2^-120 .. 2^60; and in the formats that have weights of zero, a row whose large activation meets them: what lies
    # below it by more than 2^31 counts as exactly as the rest (the next test shows that for every format)
    n, k, m = 48, 1024, 9
    wb = synth.make_weight_bytes(n, k, qtype, seed=11)
    dense = O.c_dequantize(wb, qtype).reshape(n, k).astype(np.float64)
    rng = np.random.default_rng(int(qtype))
    xb = synth.make_x(m, k, seed=1) * np.exp2(rng.integers(-120, 60, size=(m, k))).astype(np.float32)
    xb[0] = synth.make_x(1, k, seed=2)[0] * np.float32(2.0 ** -50)
    col = int(np.argmax((dense == 0).sum(0)))
    xb[0, col] = 2.0 ** 30
    xb[1] = 0
    got = product(xb, wb, qtype, n, k).numpy().astype(np.float64)
    want = xb.astype(np.float64) @ dense.T
    scale = np.abs(xb.astype(np.float64)) @ np.abs(dense).T
    assert np.all(np.abs(got - want) <= scale * 1e-5)
    zero = dense[:, col] == 0
    assert np.all(np.abs(got[0] - want[0])[zero] <= (np.abs(xb[0].astype(np.float64)) @ np.abs(dense).T)[zero] * 1e-5)
    assert not got[1].any()


@pytest.mark.skipif(not ALWAYS, reason="runs in the child process")
@pytest.mark.parametrize("qtype", FORMATS, ids=lambda t: t.name)
def test_magnitudes_far_below_the_largest_of_their_block(qtype):
    # in every batch row two neighbouring columns hold 2^30 and -2^30 and everything else is about 2^42 to 2^112 below: in the weight rows whose two
    # weights are equal the large terms cancel exactly, and what is left is the product of the small ones, the block's own among them
    n, k, m = 400, 1024, 11
    wb = synth.make_weight_bytes(n, k, qtype, seed=12)
    dense = O.c_dequantize(wb, qtype).reshape(n, k).astype(np.float64)
    pairs = np.argsort((dense[:, 0::4] == dense[:, 1::4]).sum(0))[-m:] * 4      # the pairs with the most equal weights
    xb = synth.make_x(m, k, seed=6) * np.exp2(-12.0 - 7.0 * np.arange(m))[:, None].astype(np.float32)
    small = torch.from_numpy(xb).to(torch.bfloat16).double().numpy()
    for i, c in enumerate(pairs):
        small[i, c:c + 2] = 0
        xb[i, c], xb[i, c + 1] = 2.0 ** 30, -2.0 ** 30
    got = product(xb, wb, qtype, n, k).numpy().astype(np.float64)
    want, scale = small @ dense.T, np.abs(small) @ np.abs(dense).T
    for i, c in enumerate(pairs):
        equal = dense[:, c] == dense[:, c + 1]
        assert equal.any() and np.all(np.abs(got[i] - want[i])[equal] <= scale[i][equal] * 1e-5), (i, c)
        assert np.abs(want[i])[equal].max() > 0.01 * scale[i][equal].max()      # far above the bar: a term left out shows


@pytest.mark.skipif(not ALWAYS, reason="runs in the child process")
@pytest.mark.parametrize("qtype", [QT.Q4_K, QT.Q6_K, QT.IQ4_XS, QT.IQ1_S], ids=lambda t: t.name)
def test_not_finite(qtype):
    n, k, m = 40, 1280, 11
    wb = synth.make_weight_bytes(n, k, qtype, seed=4)
    xb = synth.make_x(m, k, seed=5)
    xb[1, 700] = np.inf
    xb[2, 3] = np.nan
    xb[9, 1279] = -np.inf
    xb[10, 40] = 2.0 ** 127    # sums that leave the float32 range on the way
    dense = O.c_dequantize(wb, qtype).reshape(n, k).astype(np.float32)
    with np.errstate(all="ignore"):
        want = (xb.astype(np.float64) @ dense.T.astype(np.float64))
    got = product(xb, wb, qtype, n, k).numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf].astype(np.float32))
    fin = np.isfinite(want) & (np.abs(want) < 1e38)
    assert np.allclose(got[fin], want[fin], rtol=1e-4, atol=1e-4 * np.abs(want[:1]).max())


@pytest.mark.parametrize("qtype", [QT.Q4_K, QT.Q5_K, QT.Q6_K], ids=lambda t: t.name)
@pytest.mark.parametrize("k", [256, 1792, 2048, 2304])
def test_three_and_four_rows_around_the_column_limit(qtype, k):
    # up to 2048 columns the batch kernel takes these (Q6_K at 2048 only), above it the tiled one; the two rows beside them never
    for n in (1, 17, 300):
        wb = synth.make_weight_bytes(n, k, qtype, seed=n)
        for m in (2, 3, 4):
            xb = synth.make_x(m, k, seed=m)
            got = product(xb, wb, qtype, n, k).numpy()
            assert O.rel_l2(got, O.c_matmul(O.bf16_bits(xb), wb, qtype)) <= 2e-5, (n, k, m)
            assert np.array_equal(got.view(np.uint32), product(xb, wb, qtype, n, k).numpy().view(np.uint32))
