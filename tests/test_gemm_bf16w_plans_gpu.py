"""The bf16-weight tcgen05 GEMM (gemm_bf16w.cu) over its plans: batch tiles of 32 to 512 columns, single CTAs and pairs, a tile per CTA, clusters of 2, 4
and 8 ranges of K per tile, equal ranges that cut tiles, several segments per CTA, rows and batch ragged against every tile.

Bar: the weights are those of the decode kernel rounded once to bf16, so the float32 output differs from the float64 product of these weights by the
float32 sums alone: K = 8192 terms, each sum within 2^-24, sqrt(8192) 2^-24 = 5e-6 if they all went the same way as often as not; 1e-5.  Launches repeat
bit for bit and leave the scratch's counters at zero."""
import ctypes

import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

from gguf_jax_b200 import _lib, synth

pytestmark = pytest.mark.gpu
SHAPES = [(33, 2048, 17), (130, 2048, 65), (4700, 2048, 17), (33, 6144, 17), (9500, 2048, 17), (33, 2048, 130), (33, 2048, 200), (4700, 2048, 33),
          (9500, 2048, 33), (4700, 6144, 33), (33, 4096, 257), (33, 2048, 257), (4700, 2048, 65), (9500, 2048, 65), (4700, 8192, 65), (19000, 2048, 65),
          (33, 4096, 1100), (33, 2048, 1100), (4104, 4096, 257), (6200, 2048, 513), (130, 2048, 1100), (6200, 2048, 130), (9500, 2048, 130),
          (19000, 2048, 130), (9500, 6144, 130), (9500, 2048, 257), (9496, 2048, 1025), (20001, 6144, 257)]


@pytest.mark.parametrize("n,k,m", SHAPES, ids=str)
@pytest.mark.parametrize("qtype", [QT.Q4_K, QT.Q5_K, QT.Q6_K], ids=lambda t: t.name)
def test_plans(qtype, n, k, m, monkeypatch):
    monkeypatch.setenv("GGQ_GEMM_KERNEL", "bf16w")
    L, dev = _lib.lib(), torch.cuda.current_device()
    _lib.ensure_tables(dev)
    w = synth.make_weight_on_device(n, k, qtype, seed=n + m, device="cuda")
    x = torch.randn((m, k), device="cuda").to(torch.bfloat16)
    ws = torch.zeros(L.ggq_workspace_bytes(int(qtype), n, k, m), dtype=torch.uint8, device="cuda")

    def product(dtype, code):
        y = torch.full((m, n), float("nan"), dtype=dtype, device="cuda")
        _lib.check(L.ggq_gemm(int(qtype), w.data.data_ptr(), n, k, x.data_ptr(), m, y.data_ptr(), code, ws.data_ptr(), ws.numel(),
                              torch.cuda.current_stream().cuda_stream))
        return y

    y = product(torch.float32, _lib.GGQ_F32)
    want = x.double() @ w.dequantize(torch.bfloat16).double().T
    assert ((y.double() - want).norm() / want.norm()).item() <= 1e-5
    assert torch.equal(product(torch.float32, _lib.GGQ_F32), y)
    for dtype, code in ((torch.bfloat16, _lib.GGQ_BF16), (torch.float16, _lib.GGQ_F16)):
        assert torch.equal(product(dtype, code), y.to(dtype))
    assert not ws[128 * 1024:4 * 1024 * 1024].any()
    word = ctypes.c_int32(-1)
    assert L.ggq_read_status(dev, ctypes.byref(word)) == 0 and word.value == 0
