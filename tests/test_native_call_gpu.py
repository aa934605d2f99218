"""The native call path of `matmul` against the Python path it stands for: same results for every form of activations, and the
forms it must leave alone (gradients, host memory, transforms, subclasses, shapes and batches outside the fused route)."""
import threading
import time

import numpy as np
import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import _lib, kernels, quants, synth

pytestmark = pytest.mark.gpu


def native(x, w, force=False, budget=1 << 29):
    return _lib.native().fast_matmul(x, w.data, w.qtype, w.shape, force, budget)


@pytest.fixture(scope="module")
def weight():
    w = synth.make_weight(96, 2048, QT.Q4_K, seed=1, device="cuda")
    x = torch.randn((16, 2048), device="cuda").bfloat16()
    for m in (1, 2, 16):
        gj.matmul(x[:m], w)            # the stream's scratch
    return w, x


def test_takes_the_common_call(weight):
    w, x = weight
    for a in (x[:1], x[3], x.reshape(2, 2, 4, 2048), x[:6:2], x.T.contiguous().T[:5]):
        got = native(a, w)
        want = kernels.fused_matmul(a, w)
        assert got.shape == want.shape == (*a.shape[:-1], 96) and got.dtype == torch.bfloat16 and got.is_contiguous()
        assert torch.equal(got, want) and torch.equal(gj.matmul(a, w), want)
    with torch.inference_mode():
        assert native(x[:2], w).is_inference()
    with torch.no_grad():
        assert not native(x[:2].requires_grad_(True), w).requires_grad
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert native(x[:2], w) is None                 # no scratch on this stream yet: the Python path makes it
        first = gj.matmul(x[:2], w)
        second = native(x[:2], w)
    torch.cuda.synchronize()
    assert torch.equal(first, second) and torch.equal(first, kernels.fused_matmul(x[:2], w))


def test_leaves_everything_else_to_the_python_path(weight):
    w, x = weight

    class Sub(torch.Tensor):
        pass

    assert native(x.clone().requires_grad_(True), w) is None
    assert native(x.float(), w) is None and native(x.cpu(), w) is None
    assert native(x[:, :1024], w) is None and native(x[:0], w) is None
    assert native(x.as_subclass(Sub), w) is None
    assert native(x, synth.make_weight(96, 2048, QT.Q4_K, seed=1, device="cuda").astype(torch.float32)) is not None   # fused: w.dtype plays no part
    big = torch.randn((64, 2048), device="cuda").bfloat16()
    assert native(big, w, budget=0) is None and native(big, w, budget=4 * 96 * 2048 - 1) is None    # dense, but not in one piece here
    assert native(big, synth.make_weight(97, 2048, QT.Q8_0, seed=1, device="cuda")) is None         # rows of the result not 16-byte aligned
    for bad in (object(), None, [x]):
        assert native(bad, w) is None
    with pytest.raises(ValueError):
        gj.matmul(x[:, :1024], w)
    with pytest.raises(TypeError):
        gj.matmul(x, w.data)
    x2 = x.clone().requires_grad_(True)
    gj.matmul(x2, w).float().sum().backward()
    assert x2.grad is not None and x2.grad.shape == x2.shape


def test_dense_route_in_one_piece():
    for qtype in (QT.Q4_K, QT.Q8_0, QT.IQ3_S, QT.MXFP4):
        w = synth.make_weight(96, 2048, qtype, seed=2, device="cuda")
        x = torch.randn((2, 40, 2048), device="cuda").bfloat16()
        want = gj.dequant_matmul(x, w)
        got = native(x, w)
        assert got.shape == (2, 40, 96) and got.is_contiguous()
        assert torch.equal(got, want) and torch.equal(gj.matmul(x, w), want)
        assert gj.matmul(x, w.astype(torch.float32)).dtype == torch.float32          # another dense dtype: the Python path
    saved = quants._DEQUANT[QT.Q8_0]
    try:
        gj.register_dequant(QT.Q8_0, lambda b, d: torch.ones((b.shape[0], 32), dtype=d, device=b.device), override=True)
        w = synth.make_weight(96, 2048, QT.Q8_0, seed=2, device="cuda")
        assert torch.equal(gj.matmul(x, w), gj.dequant_matmul(x, w)) and not torch.equal(gj.matmul(x, w), native(x, w))
    finally:
        gj.register_dequant(QT.Q8_0, saved, override=True)
    assert torch.equal(gj.matmul(x, w), native(x, w))


def test_under_capture(weight):
    w, x = weight
    want = gj.matmul(x[:4], w)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        gj.matmul(x[:4], w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = gj.matmul(x[:4], w)
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_first_call_of_a_stream_under_capture_takes_no_scratch_it_can_do_without():
    w = synth.make_weight(14336, 2048, QT.Q8_0, seed=4, device="cuda")
    x = torch.randn((2, 2048), device="cuda").bfloat16()
    want = gj.matmul(x, w)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = gj.matmul(x, w)
    graph.replay()
    with torch.cuda.stream(stream):
        z = gj.matmul(x, w)
    torch.cuda.synchronize()
    assert torch.equal(z, want)
    assert ((y.double() - want.double()).norm() / want.double().norm()).item() <= 2 ** -8      # another kernel's summation order


def test_force_fused_is_any_truth_value():
    """Above the cap: the fused kernel (float32 weights) for whatever is true, the dense route (weights rounded to bf16) otherwise."""
    w = synth.make_weight(96, 2048, QT.Q8_0, seed=6, device="cuda")
    x = torch.randn((40, 2048), device="cuda").bfloat16()
    fused, dense = kernels.fused_matmul(x, w), gj.dequant_matmul(x, w)
    assert not torch.equal(fused, dense)
    for value in (True, 1, np.True_, "yes"):
        assert torch.equal(gj.matmul(x, w, force_fused=value), fused), value
    for value in (False, 0, np.False_, None):
        assert torch.equal(gj.matmul(x, w, force_fused=value), dense), value
    with pytest.raises(ValueError):
        gj.matmul(x, w, force_fused=np.array([1, 0]))


def test_two_graphs_captured_on_a_cold_stream_replay_in_any_order():
    """K-quants cannot do without scratch: each capture that finds none on its stream takes its own, cleared on every replay."""
    w = synth.make_weight(4096, 6144, QT.Q4_K, seed=7, device="cuda")
    xs = [torch.randn((m, 6144), device="cuda").bfloat16() for m in (3, 12)]
    want = [gj.matmul(x, w) for x in xs]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graphs, results = [], []
    for x in xs:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=stream):
            results.append([gj.matmul(x, w), gj.matmul(x, w)])
    with torch.cuda.stream(stream):
        eager = gj.matmul(xs[1], w)                    # before either graph has run
    torch.cuda.synchronize()
    assert torch.equal(eager, want[1])
    for i in (1, 0, 1):
        for y in results[i]:
            y.zero_()
        graphs[i].replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, want[i]) for y in results[i]), i
        assert torch.equal(gj.matmul(xs[i], w), want[i])


def test_a_graph_replays_after_the_streams_scratch_has_grown():
    small, big = synth.make_weight(4096, 6144, QT.Q4_K, seed=8, device="cuda"), synth.make_weight(8192, 28672, QT.Q4_K, seed=9, device="cuda")
    x, xb = (torch.randn((12, k), device="cuda").bfloat16() for k in (6144, 28672))
    want = gj.matmul(x, small)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        gj.matmul(x, small)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = gj.matmul(x, small)
    with torch.cuda.stream(stream):
        grown = gj.matmul(xb, big, force_fused=True)
        others = [torch.full((1 << 20,), 7, device="cuda") for _ in range(64)]         # whatever the allocator has free
        y.zero_()
        graph.replay()
        again = gj.matmul(xb, big, force_fused=True)
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(grown, again)
    assert all(bool((t == 7).all()) for t in others)


@pytest.mark.parametrize("m", [1, 40], ids=["fused", "dense"])
def test_other_threads_run_while_a_call_waits_for_the_device(m):
    """A launch waits once about a thousand are queued behind a busy kernel (a second here).  A thread that only looks at the clock
    must not be held up for that long."""
    w = synth.make_weight(96, 2048, QT.Q4_K, seed=10, device="cuda")
    x = torch.randn((m, 2048), device="cuda").bfloat16()
    gj.matmul(x, w)
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), [0.0]

    def watch():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps[0] = max(gaps[0], now - last)
            last = now

    watcher = threading.Thread(target=watch)
    watcher.start()
    start = time.perf_counter()
    torch.cuda._sleep(2_000_000_000)               # about a second at 1.9 GHz
    for _ in range(3000):
        gj.matmul(x, w)
    issued = time.perf_counter() - start
    stop.set()
    watcher.join()
    torch.cuda.synchronize()
    assert issued > 0.5, "the queue never filled: nothing was tested"
    assert gaps[0] < 0.25, gaps[0]
