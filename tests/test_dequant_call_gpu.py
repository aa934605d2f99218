"""``QuantizedArray.dequantize`` as one native call: the bits, shapes and types of the Python path for every format, and that path where the payload is
not contiguous, off alignment, of another size, on nothing that decodes, or its decoder the caller's."""
import pytest
import torch
from gguf.constants import GGML_QUANT_SIZES
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import _lib, quants, synth

pytestmark = pytest.mark.gpu


def _same(w, dtype):
    got = w.dequantize(dtype)
    want = quants.dequantize(w.data, w.qtype, dtype).reshape(w.shape)
    assert got.dtype == want.dtype and got.shape == want.shape and got.device == want.device and got.is_contiguous()
    bits = torch.int32 if dtype == torch.float32 else torch.int16
    assert torch.equal(got.view(bits), want.view(bits))
    return got


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("qtype", sorted(quants._builtins, key=lambda t: t.name), ids=lambda t: t.name)
def test_every_format(qtype, dtype):
    _lib.ensure_tables(torch.cuda.current_device())
    block, size = GGML_QUANT_SIZES[qtype]
    data = synth.make_weight_on_device(6, 2 * max(block, 32), qtype, 3, "cuda").data if block > 1 else torch.randint(0, 120, (6, 64 * size), dtype=torch.uint8,
                                                                                                                  device="cuda")
    k = data.shape[-1] // size * block
    for shape, payload in (((6, k), data), ((2, 3, k), data.reshape(2, 3, -1)), ((5, k), data[1:]), ((3, k), data[::2]),
                           ((6, k // 2) if k // 2 % block == 0 else (6, k), data[:, :data.shape[1] // 2] if k // 2 % block == 0 else data)):
        w = gj.QuantizedArray(payload, qtype, shape)
        _same(w, dtype)
    assert _lib.native().fast_dequant(data, qtype, (6, k), quants._backend.dtype_code(dtype)) is not None
    assert _lib.native().fast_dequant(data[::2], qtype, (3, k), quants._backend.dtype_code(dtype)) is None


def test_what_the_native_call_leaves_alone():
    w = synth.make_weight_on_device(8, 256, QT.Q8_0, 3, "cuda")
    fast = _lib.native().fast_dequant
    for shape in ((8, 255), (4, 256), (8, 0), (-8, -256), (1 << 40, 1 << 40), [8, 256], (8, "a")):
        assert fast(w.data, w.qtype, shape, 0) is None
    assert fast(w.data, w.qtype, w.shape, 3) is None and fast(w.data, w.qtype, w.shape, -1) is None and fast(w.data, 999, w.shape, 0) is None
    assert fast(w.data.cpu(), w.qtype, w.shape, 0) is None and fast(w.data.view(torch.int8), w.qtype, w.shape, 0) is None
    with pytest.raises(RuntimeError):
        gj.QuantizedArray(w.data, w.qtype, (4, 256)).dequantize()
    with pytest.raises(TypeError):
        w.dequantize(torch.float64)
    own = lambda blocks, dtype: torch.full((blocks.shape[0], 32), 7, dtype=dtype, device=blocks.device)     # noqa: E731
    builtin = quants._DEQUANT[QT.Q8_0]
    gj.register_dequant(QT.Q8_0, own, override=True)
    try:
        assert bool((w.dequantize() == 7).all())
    finally:
        gj.register_dequant(QT.Q8_0, builtin, override=True)
    assert not bool((w.dequantize() == 7).all())


def test_in_a_captured_graph_and_on_another_stream():
    w = synth.make_weight_on_device(64, 4096, QT.Q6_K, 3, "cuda")
    want = _same(w, torch.bfloat16)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        got = w.dequantize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            kept = w.dequantize()
        graph.replay()
    stream.synchronize()
    assert torch.equal(got, want) and torch.equal(kept, want)
