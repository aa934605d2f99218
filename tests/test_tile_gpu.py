"""The tiled fused multiply (gemv_tile.cu, every block format, batch 1..16) and what takes its place on small weights
against the CPU oracle on a B200, through the public wrappers / the C ABI.

Bars: float32 output within 2e-5 relative L2 of the oracle's double-accumulated product (i.e. nothing
but float32 summation order separates them); bf16 output within 2e-3 relative L2 and the reference's
elementwise rtol = 1e-2, atol = 1e-2 max|ref|; a one-hot activation returns the decoded weight times
the activation exactly (for activations that are powers of two), at every position of a superblock; a launch
is deterministic."""
import os

import numpy as np
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import _lib, kernels, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TILE = [QT.Q4_K, QT.Q5_K, QT.Q6_K, QT.Q2_K, QT.IQ4_XS, QT.IQ2_XXS, QT.IQ2_XS, QT.IQ2_S, QT.IQ3_XXS, QT.IQ3_S, QT.IQ1_S, QT.IQ1_M]
LOWBIT_SWEEP = [QT.Q2_K, QT.IQ1_S, QT.IQ1_M, QT.IQ2_XXS, QT.IQ2_XS, QT.IQ2_S, QT.IQ3_XXS, QT.IQ3_S, QT.IQ4_XS]


def on_device(wb, qt, n, k):
    return gj.QuantizedArray.from_bytes(wb, qt, shape=(n, k), device="cuda")


def to_x(x):
    return torch.from_numpy(x).cuda().to(torch.bfloat16)


@pytest.mark.parametrize("qtype", TILE, ids=lambda t: t.name)
def test_batches_and_ragged_shapes(qtype):
    # K multiples of 2048 keep rows 16-byte aligned for every format; N ragged against 16 and 32
    for n, k in [(200, 2048), (33, 4096), (1100, 6144)]:
        wb = synth.make_weight_bytes(n, k, qtype, seed=n)
        w = on_device(wb, qtype, n, k)
        for m in (1, 2, 3, 4, 5, 8, 9, 16):
            xb = synth.make_x(m, k, seed=m)
            ref = O.c_matmul(O.bf16_bits(xb), wb, qtype)
            got32 = kernels.fused_matmul(to_x(xb), w, out_dtype=torch.float32).cpu().numpy()
            assert O.rel_l2(got32, ref) <= 2e-5, (qtype.name, n, k, m)
            got16 = kernels.fused_matmul(to_x(xb), w).float().cpu().numpy()
            np.testing.assert_allclose(got16, ref, rtol=1e-2, atol=1e-2 * np.abs(ref).max())
            assert np.array_equal(got16, torch.from_numpy(got32).to(torch.bfloat16).float().numpy())


@pytest.mark.parametrize("qtype", TILE, ids=lambda t: t.name)
def test_one_hot_is_exact_at_every_position_of_a_superblock(qtype):
    n, k = 64, 2048
    wb = synth.make_weight_bytes(n, k, qtype, seed=7)
    w = on_device(wb, qtype, n, k)
    dense = O.ref_dequantize(wb, qtype)
    cols = list(range(256)) + [700, 1023, 1024, k - 1]
    for lo in range(0, len(cols), 8):
        sel = cols[lo:lo + 8]
        x = np.zeros((len(sel), k), dtype=np.float32)
        x[np.arange(len(sel)), sel] = 1.0
        got = kernels.fused_matmul(to_x(x), w, out_dtype=torch.float32).cpu().numpy()
        want = dense[:, sel].T.astype(np.float32)
        assert np.array_equal(got, want), (qtype.name, sel)
    x = np.zeros((1, k), dtype=np.float32)
    x[0, 77] = -4.0
    got = kernels.fused_matmul(to_x(x), w, out_dtype=torch.float32).cpu().numpy()
    assert np.array_equal(got[0], dense[:, 77] * np.float32(-4.0))


@pytest.mark.parametrize("qtype", [QT.Q4_K, QT.IQ3_S, QT.IQ1_M], ids=lambda t: t.name)
def test_activation_magnitudes(qtype):
    n, k = 96, 4096
    wb = synth.make_weight_bytes(n, k, qtype, seed=3)
    w = on_device(wb, qtype, n, k)
    base = synth.make_x(2, k, seed=3)
    for e in (-60, -20, 0, 20, 60):
        xb = base * np.float32(2.0 ** e)
        xb[1] *= np.float32(2.0 ** -7)          # the two batch rows differ in magnitude
        ref = O.c_matmul(O.bf16_bits(xb), wb, qtype)
        got = kernels.fused_matmul(to_x(xb), w, out_dtype=torch.float32).cpu().numpy()
        for r in range(2):
            assert O.rel_l2(got[r], ref[r]) <= 2e-5, (qtype.name, e, r)


@pytest.mark.parametrize("qtype", [QT.Q4_K, QT.IQ2_S], ids=lambda t: t.name)
def test_deterministic_and_row_slices_agree_with_the_whole(qtype):
    """The same launch twice gives the same bits (fixed summation order, no float atomics).  A launch on a
    row slice may cut K differently (the split adapts to the row count), so its rows agree with the
    whole-weight launch only up to float32 summation order: within 4e-6 relative to the row's scale."""
    n, k = 4096, 8192
    wb = synth.make_weight_bytes(n, k, qtype, seed=11)
    xb = synth.make_x(3, k, seed=12)
    whole = kernels.fused_matmul(to_x(xb), on_device(wb, qtype, n, k), out_dtype=torch.float32).cpu().numpy()
    again = kernels.fused_matmul(to_x(xb), on_device(wb, qtype, n, k), out_dtype=torch.float32).cpu().numpy()
    assert np.array_equal(again.view(np.uint32), whole.view(np.uint32))
    scale = np.abs(whole).max()
    for parts in (2, 8):
        rows = n // parts
        for p in (0, parts - 1):
            part = kernels.fused_matmul(to_x(xb), on_device(wb[p * rows:(p + 1) * rows], qtype, rows, k),
                                        out_dtype=torch.float32).cpu().numpy()
            np.testing.assert_allclose(part, whole[:, p * rows:(p + 1) * rows], rtol=0, atol=4e-6 * scale)


@pytest.mark.parametrize("qtype", LOWBIT_SWEEP, ids=lambda t: t.name)
def test_low_bit_sweep_shape_sampled_rows(qtype):
    """The 8192 x 28672 weight of the low-bit sweep at batch 1, 4 and 8: 256 sampled rows against the oracle.
    The relative-L2 bar on the bf16 result is applied from 512 outputs on: the output rounding alone
    contributes about 1.6e-3, so the statistic needs that many samples to sit below 2e-3 reliably."""
    n, k = 8192, 28672
    wb = synth.make_weight_bytes(n, k, qtype, seed=0)
    w = on_device(wb, qtype, n, k)
    rows = np.sort(np.random.default_rng(1).choice(n, size=256, replace=False))
    for m in (1, 4, 8):
        xb = synth.make_x(m, k, seed=m)
        ref = O.c_matmul(O.bf16_bits(xb), wb[rows], qtype)
        got32 = kernels.fused_matmul(to_x(xb), w, out_dtype=torch.float32).cpu().numpy()[:, rows]
        assert O.rel_l2(got32, ref) <= 2e-5, (qtype.name, m)
        got16 = gj.matmul(to_x(xb), w).float().cpu().numpy()[:, rows]
        if got16.size >= 512:
            assert O.rel_l2(got16, ref) <= 2e-3, (qtype.name, m)
        np.testing.assert_allclose(got16, ref, rtol=1e-2, atol=1e-2 * np.abs(ref).max())


TILE_SMALL_BLOCKS = [QT.Q8_0, QT.Q4_0, QT.Q4_1, QT.Q5_0, QT.Q5_1, QT.IQ4_NL, QT.MXFP4, QT.NVFP4, QT.Q3_K, QT.TQ1_0, QT.TQ2_0]


@pytest.mark.parametrize("qtype", TILE_SMALL_BLOCKS, ids=lambda t: t.name)
def test_formats_of_small_blocks_at_tile_edges(qtype):
    """Same bar as above (float32 sums in another order) for the legacy, FP4, ternary and Q3_K formats: one and several
    16-row tiles with and without a remainder, one superblock and several chunks, every number of passes."""
    for n, k in [(1, 2048), (16, 2048), (200, 2048), (1100, 6144), (4100, 4096)]:
        wb = synth.make_weight_bytes(n, k, qtype, seed=n)
        w = on_device(wb, qtype, n, k)
        for m in (1, 2, 3, 8, 9, 16):
            xb = synth.make_x(m, k, seed=m)
            ref = O.c_matmul(O.bf16_bits(xb), wb, qtype)
            got = kernels.fused_matmul(to_x(xb), w, out_dtype=torch.float32).cpu().numpy()
            assert O.rel_l2(got, ref) <= 2e-5, (qtype.name, n, k, m)


@pytest.mark.parametrize("n", [40, 2056])
@pytest.mark.parametrize("qtype", TILE_SMALL_BLOCKS + [QT.Q2_K, QT.IQ4_XS, QT.IQ2_XS, QT.IQ1_S], ids=lambda t: t.name)
def test_non_finite_activations_give_what_the_decoded_weights_give(qtype, n):
    """An infinite activation times the decoded weights: infinities keep their sign, and only weights that are exactly
    zero (or infinities that cancel) give NaN.  40 rows go to the MMA kernel, 2056 to the tiled one."""
    k = 2048
    wb = synth.make_weight_bytes(n, k, qtype, seed=5)
    dense = O.ref_dequantize(wb, qtype).astype(np.float32)
    xb = synth.make_x(2, k, seed=5)
    xb[1, 300] = -np.inf
    got = kernels.fused_matmul(to_x(xb), on_device(wb, qtype, n, k), out_dtype=torch.float32).cpu().numpy()
    assert np.isfinite(got[0]).all()
    want = np.where(dense[:, 300] == 0, np.nan, -np.sign(dense[:, 300]) * np.inf)
    assert np.array_equal(got[1], want, equal_nan=True), qtype.name


@pytest.mark.parametrize("exponent", [-90, 90])
@pytest.mark.parametrize("qtype", [QT.Q4_K, QT.Q5_K, QT.Q6_K], ids=lambda t: t.name)
def test_activations_far_from_one_on_small_weights(qtype, exponent):
    """Activations around 2^-90 and 2^90 at 2..4 rows: the tiled kernel scales each row by a power of two, so the result is the
    ordinary one times that power, to the same 2e-5 (the MMA kernel of the larger batches keeps about 2^-50 to 2^62)."""
    n, k = 200, 2048
    wb = synth.make_weight_bytes(n, k, qtype, seed=9)
    w = on_device(wb, qtype, n, k)
    for m in (2, 3, 4):
        xb = synth.make_x(m, k, seed=m)
        got = kernels.fused_matmul(to_x(xb) * 2.0 ** exponent, w, out_dtype=torch.float32).cpu().numpy().astype(np.float64)
        assert O.rel_l2(np.ldexp(got, -exponent), O.c_matmul(O.bf16_bits(xb), wb, qtype)) <= 2e-5, (qtype.name, m)


@pytest.mark.parametrize("qtype", [QT.Q6_K, QT.Q2_K, QT.Q3_K, QT.IQ4_XS, QT.IQ2_XXS, QT.IQ2_XS, QT.IQ2_S, QT.IQ3_XXS, QT.IQ3_S, QT.IQ1_S,
                                   QT.IQ1_M, QT.TQ1_0, QT.TQ2_0, QT.MXFP4], ids=lambda t: t.name)
def test_rows_at_every_offset_of_a_16_byte_piece(qtype):
    """K = 256 times an odd number: consecutive rows start at different offsets modulo 16 for these formats.  Enough weights
    for the tiled kernel up to batch 8 (its rule asks for 10 M), the last row tile ragged; two slices of such rows run where the
    rule is off (test_tile_small_gpu.py), other kernels take batches 9 and 16 here."""
    for n, k in [(5003, 11 * 256), (9001, 5 * 256)]:
        wb = synth.make_weight_bytes(n, k, qtype, seed=n)
        w = on_device(wb, qtype, n, k)
        rows = np.unique(np.concatenate([np.arange(40), np.random.default_rng(2).choice(n, 200), np.arange(n - 30, n)]))
        for m in (1, 2, 4, 8, 9, 16):
            xb = synth.make_x(m, k, seed=m)
            got = kernels.fused_matmul(to_x(xb), w, out_dtype=torch.float32).cpu().numpy()[:, rows]
            assert O.rel_l2(got, O.c_matmul(O.bf16_bits(xb), wb[rows], qtype)) <= 2e-5, (qtype.name, n, k, m)


def test_more_row_tiles_than_arrival_counters():
    """16252928 rows fill the counter area; a call beyond runs on the kernels without counters, also where scratch is at hand."""
    n, k, qtype = 16252928 + 40, 256, QT.TQ1_0
    w = synth.make_weight_on_device(n, k, qtype, seed=1, device="cuda")
    rows = np.unique(np.concatenate([np.arange(50), np.random.default_rng(4).choice(n, 300), np.arange(n - 90, n)]))
    wb = w.data[torch.from_numpy(rows).cuda()].cpu().numpy()
    gj.matmul(to_x(synth.make_x(2, 4096, seed=1)), synth.make_weight(4096, 4096, QT.Q4_K, seed=1, device="cuda"))      # the stream has scratch
    for m in (1, 2):
        xb = synth.make_x(m, k, seed=m)
        got = kernels.fused_matmul(to_x(xb), w, out_dtype=torch.float32)[:, torch.from_numpy(rows).cuda()].cpu().numpy()
        assert O.rel_l2(got, O.c_matmul(O.bf16_bits(xb), wb, qtype)) <= 2e-5, m


@pytest.mark.parametrize("n", [40, 2056])
@pytest.mark.parametrize("qtype", TILE_SMALL_BLOCKS + [QT.Q2_K, QT.IQ4_XS, QT.IQ2_XS, QT.IQ1_S], ids=lambda t: t.name)
def test_a_nan_activation_stays_in_its_batch_row(qtype, n):
    k, m = 2048, 9
    wb = synth.make_weight_bytes(n, k, qtype, seed=6)
    xb = synth.make_x(m, k, seed=6)
    xb[3, 1999] = xb[8, 0] = np.nan
    got = kernels.fused_matmul(to_x(xb), on_device(wb, qtype, n, k), out_dtype=torch.float32).cpu().numpy()
    assert np.isnan(got[[3, 8]]).all()
    rest = [r for r in range(m) if r not in (3, 8)]
    assert O.rel_l2(got[rest], O.c_matmul(O.bf16_bits(xb[rest]), wb, qtype)) <= 2e-5, qtype.name


def milliseconds(x, w):
    """Time of one product among twenty that are queued when the first one starts."""
    for _ in range(3):
        gj.matmul(x, w)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda._sleep(2_000_000)
    begin.record()
    for _ in range(20):
        gj.matmul(x, w)
    end.record()
    end.synchronize()
    return begin.elapsed_time(end) / 20


@pytest.mark.parametrize("qtype,n,k,m", [(QT.IQ3_S, 14336, 4096, 4), (QT.Q8_0, 14336, 4096, 16), (QT.Q4_K, 14336, 4096, 4)], ids=str)
def test_a_batch_row_that_is_not_finite_does_not_hold_up_the_others(qtype, n, k, m):
    """All outputs of a batch row with a NaN are recomputed; one lane per output took 5 to 32 times the whole product."""
    w = synth.make_weight_on_device(n, k, qtype, seed=1, device="cuda")
    x = to_x(synth.make_x(m, k, seed=1))
    bad = x.clone()
    bad[0, 77] = float("nan")
    times = [milliseconds(a, w) for a in (x, bad)]
    assert times[1] <= 3 * times[0], times


@pytest.mark.parametrize("m", [1, 4, 8])
def test_few_long_rows_are_not_left_to_few_ctas(m):
    """The same number of weights in 512 rows and in 3584: the kernels that give a CTA whole rows took 3.1 to 4.2 times as long for
    the 512, the tiled kernel takes 1.4 to 2."""
    times = []
    for n, k in ((512, 14336), (3584, 2048)):
        w = synth.make_weight_on_device(n, k, QT.IQ3_S, seed=1, device="cuda")
        times.append(milliseconds(to_x(synth.make_x(m, k, seed=1)), w))
    assert times[0] <= 2.6 * times[1], times


def microseconds_with_and_without_scratch(qtype, n, k, m):
    """ggq_gemv with the scratch that lets every kernel run, and without, which leaves the kernels that need none."""
    L = _lib.lib()
    w = synth.make_weight_on_device(n, k, qtype, seed=1, device="cuda")
    x, y = to_x(synth.make_x(m, k, seed=1)), torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(L.ggq_scratch_bytes(int(qtype), n, k, m), dtype=torch.uint8, device="cuda")
    _lib.ensure_tables(0)
    best = [float("inf")] * 2
    for _ in range(6):
        for i, scratch in enumerate(((ws.data_ptr(), ws.numel()), (None, 0))):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(1_000_000)
            begin.record()
            for _ in range(40):
                _lib.check(L.ggq_gemv(int(qtype), w.data.data_ptr(), n, k, x.data_ptr(), m, y.data_ptr(), _lib.GGQ_BF16, *scratch,
                                      torch.cuda.current_stream().cuda_stream))
            end.record()
            end.synchronize()
            best[i] = min(best[i], begin.elapsed_time(end) * 25)
    return best


@pytest.mark.skipif(os.environ.get("GGQ_TILE_ALWAYS") == "1", reason="about the size rule, which is off")
@pytest.mark.parametrize("qtype,n,k,m", [(QT.Q6_K, 512, 1024, 2), (QT.Q6_K, 512, 1024, 4), (QT.Q6_K, 1024, 5 * 256, 3),
                                         (QT.Q6_K, 16384, 3 * 256, 5)], ids=str)
def test_scratch_does_not_slow_small_calls_down(qtype, n, k, m):
    """Weights with unaligned rows that are small, or whose rows are short, took the tiled and the batch-major kernel, up to twice
    the time of the MMA kernel, where scratch was at hand."""
    with_scratch, without = microseconds_with_and_without_scratch(qtype, n, k, m)
    assert with_scratch <= 1.15 * without, (with_scratch, without)


@pytest.mark.parametrize("m", [5, 8])
def test_q8_0_keeps_the_tiled_kernel_on_large_weights(m):
    """Its ring of copied blocks fits next to eight staged batch rows also where K is cut into chunks of eight superblocks."""
    n, k = 8192, 12288
    with_scratch, without = microseconds_with_and_without_scratch(QT.Q8_0, n, k, m)
    assert with_scratch <= 0.85 * without, (with_scratch, without)
    wb = synth.make_weight_bytes(n, k, QT.Q8_0, seed=m)
    rows = np.sort(np.random.default_rng(3).choice(n, size=64, replace=False))
    xb = synth.make_x(m, k, seed=m)
    got = kernels.fused_matmul(to_x(xb), on_device(wb, QT.Q8_0, n, k), out_dtype=torch.float32).cpu().numpy()[:, rows]
    assert O.rel_l2(got, O.c_matmul(O.bf16_bits(xb), wb[rows], QT.Q8_0)) <= 2e-5
