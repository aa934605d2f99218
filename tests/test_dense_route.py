"""The materializing route's choice between products written in place and the general way, on the CPU: a registered decoder makes
dense weights there, so that autocast, transforms, traces and modes can be tried without a device.  The in-place products
and the padded rows must be indistinguishable from one product of the whole dense weight."""
import gguf
import numpy as np
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import _matmul as mm
from gguf_jax_b200 import quants, synth

K = 128
IN_SLABS = 4 * K * 32           # a budget of 32 rows


@pytest.fixture(autouse=True)
def decoder_on_the_cpu():
    saved = quants._DEQUANT[QT.Q8_0]

    def decode(blocks, dtype):
        return torch.from_numpy(np.asarray(gguf.quants.dequantize(blocks.numpy(), QT.Q8_0))).to(dtype)

    gj.register_dequant(QT.Q8_0, decode, override=True)
    yield
    gj.register_dequant(QT.Q8_0, saved, override=True)


def case(n, m=6, seed=1):
    w = synth.make_weight(n, K, QT.Q8_0, seed=seed, device="cpu")
    return w, torch.randn((m, K), generator=torch.Generator().manual_seed(seed))


# one slab; several slabs; one slab whose rows are padded (the size rule set aside)
FORMS = [(96, None, False), (96, IN_SLABS, False), (100, IN_SLABS, False), (100, None, True)]


@pytest.mark.parametrize("n,budget,padded", FORMS)
@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("x_dtype,cast_to", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float16)], ids=str)
def test_autocast_decides_the_dtype_whatever_the_shape(n, budget, padded, train, x_dtype, cast_to, monkeypatch):
    if padded:
        monkeypatch.setattr(mm, "_PAD_FROM_OPS", 0)
    w, x = case(n)
    x = x.to(x_dtype).requires_grad_(train)
    with torch.autocast("cpu", dtype=cast_to):
        y = gj.dequant_matmul(x, w, block_bytes=budget)
        want = torch.matmul(x.detach(), w.dequantize().T)
    assert want.dtype == cast_to and y.dtype == cast_to
    assert torch.allclose(y.float(), want.float(), rtol=2 ** -7, atol=2 ** -7 * want.abs().max().item())


class Recorder(torch.overrides.TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


def test_function_modes_see_the_operations(monkeypatch):
    w, x = case(96)
    with Recorder() as mode:
        y = gj.dequant_matmul(x, w, block_bytes=IN_SLABS)
    assert torch.matmul in mode.seen and torch.mm not in mode.seen
    assert torch.allclose(y, x @ w.dequantize(torch.float32).T, rtol=2 ** -7, atol=0.1)
    # the native call path has no operations a mode could see: it is not asked, except under the mode that only sets the device
    monkeypatch.setattr(mm, "_native_matmul", lambda *a: "native")
    with Recorder(), pytest.raises(RuntimeError):
        gj.matmul(x, w)                       # the general path, which refuses host memory
    assert gj.matmul(x, w) == "native"
    with torch.device("cpu"):
        assert gj.matmul(x, w) == "native"
        with Recorder(), pytest.raises(RuntimeError):
            gj.matmul(x, w)


class Dispatched(torch.utils._python_dispatch.TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("n,budget,padded", FORMS)
def test_transforms_traces_and_modes_take_the_general_way(n, budget, padded, monkeypatch):
    """Each of these fails, or computes something else, where a product is written into its columns of the result: there is no
    batching rule and no derivative for a product with ``out=``, and a mode sees another operation."""
    if padded:
        monkeypatch.setattr(mm, "_PAD_FROM_OPS", 0)
    w, x = case(n)
    x = x.double()
    dense = w.dequantize().double()
    product = lambda a: gj.dequant_matmul(a, w, block_bytes=budget)
    assert torch.allclose(product(x), x @ dense.T)
    rows = torch.stack([x, 2 * x, -x])
    assert torch.allclose(torch.func.vmap(product)(rows), rows @ dense.T)
    assert torch.allclose(torch.func.vmap(product, in_dims=1, out_dims=1)(rows), rows @ dense.T)
    t = torch.randn_like(x)
    with torch.autograd.forward_ad.dual_level():
        y = torch.autograd.forward_ad.unpack_dual(product(torch.autograd.forward_ad.make_dual(x, t)))
    assert torch.allclose(y.primal, x @ dense.T) and torch.allclose(y.tangent, t @ dense.T)
    traced = torch.jit.trace(product, (x,), check_trace=False)
    assert torch.allclose(traced(3 * t), 3 * t @ dense.T)
    with Dispatched() as mode:
        y = product(x)
    assert torch.ops.aten.mm.out not in mode.seen and torch.ops.aten.mm.default in mode.seen
    assert torch.allclose(y, x @ dense.T)


@pytest.mark.parametrize("x_dtype,w_dtype,slabs", [
    (torch.bfloat16, torch.bfloat16, 1), (torch.float16, torch.float16, 1),      # multiplied as decoded: 2 bytes a weight
    (torch.float32, torch.bfloat16, 2), (torch.float16, torch.bfloat16, 2), (torch.bfloat16, torch.float16, 2),    # converted as well
    (torch.bfloat16, torch.float32, 2), (torch.float32, torch.float32, 2)], ids=str)
def test_slabs_are_costed_at_what_they_take(x_dtype, w_dtype, slabs, monkeypatch):
    """Weights of 64 rows where 32 fit at 4 bytes a weight: under the default budget whole where the GEMM reads the decoded copy itself;
    under autocast, where the number of rows is no multiple of 8 and under a budget that somebody set, at 4 bytes as ever."""
    calls = []
    decode = quants._DEQUANT[QT.Q8_0]
    monkeypatch.setitem(quants._DEQUANT, QT.Q8_0, lambda blocks, dtype: (calls.append(len(blocks)), decode(blocks, dtype))[1])

    def decoded(n, **kw):
        calls.clear()
        w, x = case(n)
        x = x.to(x_dtype)
        y = gj.dequant_matmul(x, w.astype(w_dtype), **kw)
        dense = w.astype(w_dtype).dequantize()
        del calls[-1]
        assert torch.allclose(y.double(), x.double() @ dense.double().T, rtol=2 ** -7, atol=0.2)
        return len(calls)

    monkeypatch.setattr(mm, "DEQUANT_BLOCK_BYTES", IN_SLABS)
    assert decoded(64) == 2 and decoded(64, block_bytes=IN_SLABS) == 2
    monkeypatch.setattr(mm, "_DEFAULT_BLOCK_BYTES", IN_SLABS, raising=False)
    assert decoded(64) == slabs and decoded(64, block_bytes=IN_SLABS) == 2
    assert decoded(68) >= 3                      # one row more than two slabs of 32 take; never in one
    with torch.autocast("cpu", dtype=torch.bfloat16):
        assert decoded(64) == 2
