"""A split-K scratch that grows while others use it: a launch of another thread on the same stream, or a captured graph."""
import ctypes
import threading
import weakref

import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import api, synth

pytestmark = pytest.mark.gpu
K, N, QC = 1024, 1024, 256


@pytest.fixture(scope="module")
def layer():
    return synth.make_layer(K, N, QC, 128, seed=3, keep_dequantized=False).to(torch.device("cuda", 0))


def _mul(layer, a):
    c = torch.zeros((a.shape[0], N), dtype=torch.float16, device=a.device)
    workspace = torch.zeros(N // 128 * 16, dtype=torch.int32, device=a.device)
    fm.mul(a, layer.B, c, layer.s, workspace, QC, group_size=128, layout="b200")
    return c


def _bind(mul_address):
    api._call.bind(mul_address, *(ctypes.cast(getattr(api.lib, f), ctypes.c_void_p).value for f in ("fp6m_mul_fused", "fp6m_mul_scratch_bytes")))


def test_scratch_of_a_launch_under_way_outlives_growth(layer):
    """A host function in the place of fp6m_mul (nothing is launched) stands for a launch that waits for room in the GPU's queue:
    meanwhile another thread grows the scratch of the same stream."""
    dev = layer.B.device
    stream = torch.cuda.Stream(dev)
    seen = []
    with torch.cuda.stream(stream):
        a = synth.make_activations(1, K, 1).to(dev)
        _mul(layer, a)                               # creates the stream's scratch
        first = api._device_buffers(dev, (1, N, K, QC))[1]
        alive, address, size = weakref.ref(first), first.data_ptr(), first.numel()
        del first

        def grow():
            with torch.cuda.stream(stream):
                seen.append(api._device_buffers(dev, (128, 8192, 8192, QC))[1])

        def stand_in(*args):
            thread = threading.Thread(target=grow)
            thread.start()
            thread.join()
            seen.append((args[9], args[10], alive() is not None))      # scratch, its size
            return 0

        prototype = ctypes.CFUNCTYPE(*([api.lib.fp6m_mul.restype] + list(api.lib.fp6m_mul.argtypes)))
        callback = prototype(stand_in)
        _bind(ctypes.cast(callback, ctypes.c_void_p).value)
        try:
            _mul(layer, a)
        finally:
            _bind(ctypes.cast(api.lib.fp6m_mul, ctypes.c_void_p).value)
    stream.synchronize()
    assert seen[0].numel() > size
    assert seen[1] == (address, size, True)


def test_one_stream_two_threads(layer):
    """One thread repeats a small call, the other asks for more scratch every time: the results of one thread alone."""
    dev = layer.B.device
    stream = torch.cuda.Stream(dev)
    small = synth.make_activations(5, K, 2).to(dev)
    growing = [synth.make_activations(m, K, m).to(dev) for m in (9, 17, 40, 100, 300)]
    with torch.cuda.stream(torch.cuda.Stream(dev)):
        ordered = fm.set_ordered_sums(True)
        want = [_mul(layer, a) for a in [small] + growing]
    results, failures = {}, []
    torch.cuda.synchronize()

    def work(name, inputs):
        try:
            with torch.cuda.stream(stream):
                results[name] = [_mul(layer, a) for a in inputs]
        except Exception as e:
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=("small", [small] * 100)), threading.Thread(target=work, args=("growing", growing * 3))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    fm.set_ordered_sums(ordered)
    assert not failures, failures
    assert all(torch.equal(c, want[0]) for c in results["small"])
    assert all(torch.equal(c, want[1 + i % len(growing)]) for i, c in enumerate(results["growing"]))
    assert fm.device_status(dev) == 0


def test_captured_graph_keeps_its_scratch(layer):
    """A graph is captured, then a larger eager call grows the stream's scratch and others allocate: the graph still replays right
    and writes to nobody else's memory."""
    dev = layer.B.device
    stream = torch.cuda.Stream(dev)
    with torch.cuda.stream(stream):
        a, large = synth.make_activations(3, K, 4).to(dev), synth.make_activations(300, K, 5).to(dev)
        want = _mul(layer, a)
        size = api._device_buffers(dev, (3, N, K, QC))[1].numel()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            c = _mul(layer, a)
        _mul(layer, large)
        others = [torch.full((size,), 0x5A, dtype=torch.uint8, device=dev) for _ in range(8)]
        for _ in range(3):
            c.zero_()
            graph.replay()
            assert torch.equal(c, want)
    torch.cuda.synchronize()
    assert all(bool((o == 0x5A).all()) for o in others)
    assert fm.device_status(dev) == 0


@pytest.mark.parametrize("attempt", range(3))
def test_first_calls_of_threads_on_one_stream(layer, attempt):
    """Nobody has made the stream's scratch when eight threads call at once, with rows that need scratches of four sizes."""
    dev = layer.B.device
    rows = [1, 8, 16, 20, 33, 64, 100, 300]
    inputs = [synth.make_activations(m, K, m).to(dev) for m in rows]
    ordered = fm.set_ordered_sums(True)
    want = [_mul(layer, a) for a in inputs]
    stream, go = torch.cuda.Stream(dev), threading.Barrier(len(rows))
    torch.cuda.synchronize()
    results, failures = {}, []

    def work(i):
        try:
            with torch.cuda.stream(stream):
                go.wait()
                results[i] = [_mul(layer, inputs[i]) for _ in range(5)]
        except Exception as e:
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(rows))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    fm.set_ordered_sums(ordered)
    assert not failures, failures
    assert all(torch.equal(c, want[i]) for i in results for c in results[i])
    assert fm.device_status(dev) == 0
