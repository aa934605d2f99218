"""Which way a call of `matmul` goes: up to `fused_batch_limit` the fused kernels multiply, whatever dtype the weight decodes to and whoever
decodes it, and their result is bfloat16; above, the dense copy."""
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import kernels, quants, synth

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
