"""Which way a call of `matmul` goes: up to `fused_batch_limit` the fused kernels multiply, whatever dtype the weight decodes to and whoever
decodes it, and their result is bfloat16; above, the dense copy.  And which of the fused kernels takes it."""
import numpy as np
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import kernels, quants, synth
from oracle import oracle as O
from tests.launched import kernels_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qtype,n,k,batches", [(QT.Q4_K, 6144, 6144, (33, 65, 256)), (QT.Q5_K, 8192, 8192, (193, 256)),
                                               (QT.Q6_K, 4096, 4096, (33, 256)), (QT.Q6_K, 14336, 4096, (257, 512))], ids=str)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=str)
def test_fused_up_to_the_limit(qtype, n, k, batches, dtype):
    w = synth.make_weight_on_device(n, k, qtype, seed=1, device="cuda").astype(dtype)
    assert gj.fused_batch_limit(w) == batches[-1]
    x = torch.randn((batches[-1] + 1, k), device="cuda").to(torch.bfloat16)
    for m in batches:
        for _ in range(2):              # the Python path, which makes the scratch, and the native one
            y = gj.matmul(x[:m], w)
            assert y.dtype == torch.bfloat16 and torch.equal(y, kernels.fused_matmul(x[:m], w)), m
    y = gj.matmul(x, w)
    assert y.dtype == torch.promote_types(dtype, torch.bfloat16) and torch.equal(y, gj.dequant_matmul(x, w))


def test_a_registered_decoder_serves_the_dense_route_only():
    w = synth.make_weight_on_device(4096, 4096, QT.Q6_K, seed=2, device="cuda")
    x = torch.randn((100, 4096), device="cuda").to(torch.bfloat16)
    saved, calls = quants._DEQUANT[QT.Q6_K], []

    def decode(blocks, dtype):
        calls.append(blocks.shape)
        return saved(blocks, dtype)

    gj.register_dequant(QT.Q6_K, decode, override=True)
    try:
        assert torch.equal(gj.matmul(x, w), kernels.fused_matmul(x, w)) and not calls
        gj.dequant_matmul(x, w)
        assert len(calls) == 1
    finally:
        gj.register_dequant(QT.Q6_K, saved, override=True)


# the batch kernel's formats but the K-quants
LOWBIT = [QT.Q2_K, QT.Q3_K, QT.IQ4_XS, QT.IQ2_XXS, QT.IQ2_XS, QT.IQ2_S, QT.IQ3_XXS, QT.IQ3_S, QT.IQ1_S, QT.IQ1_M, QT.TQ1_0, QT.TQ2_0]


@pytest.mark.parametrize("qtype,n,k,m", [(qt, 600_011, 256, 16) for qt in LOWBIT + [QT.Q4_K, QT.Q5_K, QT.Q6_K]] +
                         [(QT.IQ3_S, 256_000, 2048, 9), (QT.Q2_K, 1_300_003, 256, 5)], ids=str)
def test_weights_of_very_many_rows_are_cut(qtype, n, k, m):
    """Too many rows for one launch of the batch kernel, which keeps every tile's sums: parts of rows, each multiplied by it, and the
    outputs that are not finite computed again in every part.  Same bar as for one launch (test_batch_gpu.py)."""
    w = synth.make_weight_on_device(n, k, qtype, seed=3, device="cuda")
    xb = synth.make_x(m, k, seed=m)
    xb[1, 3] = np.inf
    x = torch.from_numpy(xb).cuda().to(torch.bfloat16)
    product = lambda: kernels.fused_matmul(x, w, out_dtype=torch.float32)
    names = kernels_of(product)
    assert 2 <= len(names) <= 4 and all("gemv_batch_kernel" in name for name in names), names
    # the first and last rows, the tiles around every place where the parts may meet, and some rows between
    tiles = -(-n // 16)
    cuts = [16 * -(-tiles // parts) * i for parts in (2, 3, 4) for i in range(1, parts)]
    pick = np.unique(np.clip(np.concatenate([np.arange(16), *[c + np.arange(-17, 18) for c in cuts], n - 1 - np.arange(17),
                                             np.random.default_rng(0).integers(0, n, 64)]), 0, n - 1))
    rows = w.data[torch.from_numpy(pick).cuda()].cpu().numpy()
    got = product()[:, torch.from_numpy(pick).cuda()].cpu().numpy()
    fine = np.arange(m) != 1
    assert O.rel_l2(got[fine], O.c_matmul(O.bf16_bits(xb[fine]), rows, qtype)) <= 2e-5
    column = O.c_dequantize(rows, qtype).reshape(len(pick), k)[:, 3]
    assert np.array_equal(np.isnan(got[1]), column == 0)
    assert np.array_equal(got[1][column != 0], np.sign(column[column != 0]) * np.inf)


@pytest.mark.parametrize("qtype,n,k,m,kernel", [
    # Q6_K from 9 rows on: the batch-major kernel from a number of weights on that falls with the columns
    (QT.Q6_K, 8192, 20480, 9, "wide"), (QT.Q6_K, 8192, 20480, 8, "batch"), (QT.Q6_K, 4096, 16384, 16, "batch"), (QT.Q6_K, 20480, 10240, 16, "wide"),
    (QT.Q6_K, 32000, 8192, 16, "wide"), (QT.Q6_K, 28672, 8192, 9, "batch"), (QT.Q6_K, 65536, 4096, 16, "batch"),
    (QT.Q6_K, 8000, 20736, 16, "wide"), (QT.Q6_K, 12291, 9472, 9, "wide"), (QT.Q6_K, 4096, 14592, 16, "batch"), (QT.Q6_K, 16384, 7424, 16, "batch"),
    (QT.Q5_K, 8192, 20480, 16, "batch"),
    # 9 rows and more of the low-bit formats with one row tile per SM
    (QT.IQ4_XS, 2048, 5120, 9, "mma"), (QT.Q2_K, 2368, 4608, 16, "mma"), (QT.TQ1_0, 1025, 4608, 9, "mma"), (QT.TQ1_0, 1024, 4608, 9, "batch"),
    (QT.IQ4_XS, 2369, 4608, 16, "batch"), (QT.IQ4_XS, 2048, 5632, 9, "batch"), (QT.IQ4_XS, 2048, 5120, 8, "batch"), (QT.Q6_K, 2048, 5120, 9, "batch"),
    # 3 and 4 rows of the low-bit formats: the batch kernel where there are rows enough, for IQ4_XS up to a size
    (QT.IQ3_S, 16384, 8192, 4, "batch"), (QT.IQ4_XS, 16384, 8192, 3, "tile"), (QT.IQ4_XS, 32000, 4096, 4, "tile"),
    (QT.IQ4_XS, 18432, 4608, 4, "batch"), (QT.IQ4_XS, 16384, 8192, 5, "batch"),
], ids=str)
def test_kernel_of_a_call(qtype, n, k, m, kernel):
    w = synth.make_weight_on_device(n, k, qtype, seed=4, device="cuda")
    xb = synth.make_x(m, k, seed=m)
    x = torch.from_numpy(xb).cuda().to(torch.bfloat16)
    product = lambda: kernels.fused_matmul(x, w, out_dtype=torch.float32)
    names = kernels_of(product)
    assert any(f"gemv_{kernel}" in name for name in names), names
    pick = torch.from_numpy(np.random.default_rng(0).choice(n, size=48, replace=False)).cuda()
    assert O.rel_l2(product()[:, pick].cpu().numpy(), O.c_matmul(O.bf16_bits(xb), w.data[pick].cpu().numpy(), qtype)) <= 2e-5
