"""The gradient in ``x`` of a product with a weight whose number of rows is no multiple of 8, with the contraction cut at the last multiple: the same
gradient as one product with the dense weight, in one slab and in several, in every type, under autocast and vmap, and differentiable again.  On the CPU, with a
registered decoder, and on the device with its own.

Bar: a float32 sum of at most 2445 terms against float64, 2445 half steps of 2^-24 of the largest sum of magnitudes, far more than it needs; types of 16 bits one
rounding of the result, and one each of the slabs' products and of their addends, whose magnitudes add up to the sum of magnitudes at most."""
import gguf
import numpy as np
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import _matmul as mm
from gguf_jax_b200 import quants, synth

K = 128


@pytest.fixture
def weight(monkeypatch):
    saved = quants._DEQUANT[QT.Q8_0]
    gj.register_dequant(QT.Q8_0, lambda blocks, dtype: torch.from_numpy(np.asarray(gguf.quants.dequantize(blocks.numpy(), QT.Q8_0))).to(dtype), override=True)
    monkeypatch.setattr(mm, "_CUT_FROM_OPS", 0)
    yield lambda n: synth.make_weight(n, K, QT.Q8_0, seed=n, device="cpu")
    gj.register_dequant(QT.Q8_0, saved, override=True)


def _close(got, g, dense, step):
    want, size = g.double() @ dense.double(), g.double().abs() @ dense.double().abs()
    bar = dense.shape[0] * 2.0 ** -24 * size + step / 2 * (want.abs() + 2 * size)
    assert bool(((got.double() - want).abs() <= bar).all())


@pytest.mark.parametrize("dtype,step", [(torch.float32, 0.0), (torch.bfloat16, 2.0 ** -7), (torch.float16, 2.0 ** -10)], ids=str)
@pytest.mark.parametrize("n,rows", [(3, None), (8, None), (13, None), (97, None), (100, None), (99, 33), (100, 25), (70, 7)])
def test_matches_the_dense_weight(weight, dtype, step, n, rows):
    w = weight(n).astype(dtype)
    x = torch.randn(5, K, generator=torch.Generator().manual_seed(1)).to(dtype).requires_grad_()
    g = torch.randn(5, n, generator=torch.Generator().manual_seed(2)).to(dtype)
    y = gj.dequant_matmul(x, w, block_bytes=None if rows is None else 4 * K * rows)
    (dx,) = torch.autograd.grad(y, x, g)
    assert dx.dtype == dtype and dx.shape == x.shape
    _close(dx, g, w.dequantize(), step)


def test_autocast_vmap_and_a_second_derivative(weight):
    w = weight(100).astype(torch.float32)
    dense, g = w.dequantize(), torch.randn(3, 5, 100)
    got = torch.vmap(lambda v: mm._input_cotangent(v, w, 1))(g)
    assert torch.allclose(got, g @ dense, rtol=1e-4, atol=1e-3)
    with torch.autocast("cpu", dtype=torch.bfloat16):
        a, b = mm._input_cotangent(g[0], w, 1), torch.matmul(g[0], dense)
    assert a.dtype == b.dtype and torch.allclose(a.float(), b.float(), rtol=2 ** -6, atol=2 ** -6 * b.abs().max().item())
    gg = g[0].clone().requires_grad_()
    mm._input_cotangent(gg, w, 1).square().sum().backward()
    assert torch.allclose(gg.grad, 2 * (g[0] @ dense) @ dense.T, rtol=1e-3, atol=1e-1)


@pytest.mark.gpu
@pytest.mark.parametrize("qtype,n,k,m", [(QT.Q4_0, 3001, 4672, 600), (QT.Q8_0, 9001, 2080, 257)], ids=str)
def test_the_product_itself_on_the_device(qtype, n, k, m):
    assert 2 * n * k * m >= mm._PAD_FROM_OPS
    w = synth.make_weight_on_device(n, k, qtype, seed=3, device="cuda")
    x = torch.randn((m, k), device="cuda").to(torch.bfloat16)
    y = gj.matmul(x, w)
    assert y.shape == (m, n) and y.is_contiguous()
    _close(y, x, w.dequantize().T, 2.0 ** -7)


@pytest.mark.gpu
@pytest.mark.parametrize("qtype,n,k,m,rows", [(QT.Q4_K, 2445, 1792, 1024, None), (QT.Q4_0, 2445, 1824, 1024, None), (QT.IQ2_XXS, 2442, 1792, 1200, 1221)], ids=str)
def test_on_the_device(qtype, n, k, m, rows):
    assert 2 * n * k * m >= mm._CUT_FROM_OPS
    w = synth.make_weight_on_device(n, k, qtype, seed=3, device="cuda")
    x = torch.randn((m, k), device="cuda").to(torch.bfloat16).requires_grad_()
    g = torch.randn((m, n), device="cuda").to(torch.bfloat16)
    (dx,) = torch.autograd.grad(gj.matmul(x, w, block_bytes=None if rows is None else 4 * k * rows), x, g)
    _close(dx, g, w.dequantize(), 2.0 ** -7)
