"""The materializing route: products written straight into the result and rows padded to 16 bytes give what the plain
product of the dense weight gives, at row counts that are no multiple of 8 and with slabs, and transforms take the general way.
Bars: bf16 results of float32 sums that may be taken in another order, one bf16 rounding apart at most (2^-8 relative, and
2^-9 / sqrt(3) in the 2-norm for each of the two sides)."""
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("n", [8, 9, 100, 247, 256])
@pytest.mark.parametrize("slab_rows", [None, 64, 24, 5])
def test_products_and_gradients_of_any_row_count(n, slab_rows):
    k, m = 512, 37
    w = synth.make_weight(n, k, QT.Q5_1, seed=n, device="cuda")
    budget = None if slab_rows is None else 4 * k * slab_rows
    x = torch.randn((m, k), device="cuda").bfloat16()
    dense = w.dequantize()
    y = gj.dequant_matmul(x, w, block_bytes=budget)
    assert y.shape == (m, n) and y.is_contiguous() and y.dtype == torch.bfloat16
    assert rel(y, x.double() @ dense.double().T) <= 2 ** -8
    for dtype in (torch.float32, torch.float16):
        z = gj.dequant_matmul(x.to(dtype), w, block_bytes=budget)
        want = x.to(torch.promote_types(dtype, torch.bfloat16)).double() @ dense.double().T
        assert z.dtype == torch.promote_types(dtype, torch.bfloat16) and rel(z, want) <= 1e-3
    xg = x.clone().requires_grad_(True)
    g = torch.randn((m, n), device="cuda").bfloat16()
    (dx,) = torch.autograd.grad(gj.dequant_matmul(xg, w, block_bytes=budget), xg, g)
    assert rel(dx, g.double() @ dense.double()) <= 2 ** -8
    assert gj.dequant_matmul(x[:0], w, block_bytes=budget).shape == (0, n)


def test_padded_rows_of_a_large_product():
    """Enough operations for the padded rows of the result and of the gradient."""
    m, n, k = 2048, 2049, 4096
    w = synth.make_weight(n, k, QT.Q5_1, seed=1, device="cuda")
    dense = w.dequantize()
    x = torch.randn((m, k), device="cuda").bfloat16().requires_grad_(True)
    g = torch.randn((m, n), device="cuda").bfloat16()
    y = gj.dequant_matmul(x, w, block_bytes=None)
    (dx,) = torch.autograd.grad(y, x, g)
    assert y.shape == (m, n) and y.is_contiguous()
    assert rel(y, x.double() @ dense.double().T) <= 2 ** -8 and rel(dx, g.double() @ dense.double()) <= 2 ** -8


def test_transforms_take_the_general_way():
    w = synth.make_weight(100, 512, QT.Q5_1, seed=3, device="cuda")
    x = torch.randn((4, 6, 512), device="cuda")
    dense = w.dequantize().float()
    budget = 4 * 512 * 32
    for block_bytes in (None, budget):              # one slab; several, which plain tensors have written in place
        mapped = torch.func.vmap(lambda a: gj.dequant_matmul(a, w, block_bytes=block_bytes))(x)
        assert rel(mapped, x @ dense.T) <= 1e-5
    assert rel(gj.dequant_matmul(x, w, block_bytes=budget), x @ dense.T) <= 1e-5


@pytest.mark.parametrize("case", ["float32 x", "autocast", "gradient", "bfloat16"])
def test_memory_of_a_large_weight(case):
    """20480 x 8192: 672 MB at 4 bytes a weight, the default budget 537 MB.  Alive at once is one bf16 slab (336 MB whole), and where it is
    converted its copy: two slabs then, 168 MB each and 336 (to float32) or 168 (to float16) MB more."""
    n, k, m = 20480, 8192, 64
    w = synth.make_weight_on_device(n, k, QT.Q8_0, seed=1, device="cuda")
    x = torch.randn((m, k), device="cuda").to(torch.bfloat16)
    dtype = torch.float32 if case in ("float32 x", "gradient") else torch.bfloat16
    x = x.to(dtype).requires_grad_(case == "gradient")
    gj.matmul(x[:, :k], w)                  # the library's workspace
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    with torch.autocast("cuda", dtype=torch.float16, enabled=case == "autocast"):
        y = gj.matmul(x, w)
    if case == "gradient":
        torch.autograd.grad(y, x, y.detach())
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - base <= 560 << 20
