"""Launches whose CTAs share a row group's sums, at the lines where that begins and ends: the batch-1 kernels of Q4_K, Q5_K and Q6_K (row groups whole
or cut, the last one ragged) and the batch-major kernel (activations staged by the launch itself or by a kernel before it, one contributor to 56,
columns of any magnitude, copies by tensor map and by thread).

Bar: codes and scales are exact, so the float32 output differs from the float64 product of the decoded weights by float32 sums alone: 14336 terms within
2^-24 each, sqrt(14336) 2^-24 = 7e-6 if they went the same way as often as not; 1e-5 of a column's norm.  Launches repeat bit for bit and leave the
scratch's counters at zero."""
import ctypes

import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

from gguf_jax_b200 import _lib, synth

pytestmark = pytest.mark.gpu
K_QUANTS = [QT.Q4_K, QT.Q5_K, QT.Q6_K]


def _check(qtype, n, k, m, entry, x):
    L, dev = _lib.lib(), torch.cuda.current_device()
    w = synth.make_weight_on_device(n, k, qtype, seed=n + k + m, device="cuda")
    ws = torch.zeros(max(L.ggq_workspace_bytes(int(qtype), n, k, m), L.ggq_scratch_bytes(int(qtype), n, k, m)), dtype=torch.uint8, device="cuda")

    def product():
        y = torch.full((m, n), float("nan"), device="cuda")
        _lib.check(getattr(L, entry)(int(qtype), w.data.data_ptr(), n, k, x.data_ptr(), m, y.data_ptr(), _lib.GGQ_F32, ws.data_ptr(), ws.numel(),
                                     torch.cuda.current_stream().cuda_stream))
        return y

    y, want = product(), x.double() @ w.dequantize(torch.float32).double().T
    off = (y.double() - want).norm(dim=1) / want.norm(dim=1)
    assert off.max().item() <= 1e-5, off
    assert torch.equal(product(), y)
    assert not ws[128 * 1024:4 * 1024 * 1024].any()
    word = ctypes.c_int32(-1)
    assert L.ggq_read_status(dev, ctypes.byref(word)) == 0 and word.value == 0


@pytest.mark.parametrize("n,k", [(33, 2048), (1024, 8192), (2048, 8192), (4096, 4096), (4096, 8192), (4097, 14336), (5003, 8192), (4736, 6144), (4737, 6144),
                                 (9500, 6144), (14336, 4096)], ids=str)
@pytest.mark.parametrize("qtype", K_QUANTS, ids=lambda t: t.name)
def test_one_row(qtype, n, k):
    _check(qtype, n, k, 1, "ggq_gemv", torch.randn((1, k), device="cuda").to(torch.bfloat16))


@pytest.mark.parametrize("n,k", [(33, 256), (33, 2048), (300, 14336), (1024, 4096), (2000, 5888), (4096, 4096), (9472, 2048), (9600, 2048), (4737, 4096),
                                 (9500, 4096)], ids=str)
@pytest.mark.parametrize("m", [5, 12, 17, 32])
@pytest.mark.parametrize("tma", ["1", "0"], ids=["boxes", "copies"])
@pytest.mark.parametrize("qtype", K_QUANTS, ids=lambda t: t.name)
def test_batch_major(qtype, tma, m, n, k, monkeypatch):
    monkeypatch.setenv("GGQ_GEMM_KERNEL", "wide")
    monkeypatch.setenv("GGQ_WIDE_TMA", tma)
    x = torch.randn((m, k), device="cuda") * torch.exp2(torch.linspace(-60, 60, m, device="cuda"))[:, None]
    x[0, :k // 2] = 0
    _check(qtype, n, k, m, "ggq_gemm", x.to(torch.bfloat16))
