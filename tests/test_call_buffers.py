"""The buffers that calls of `mul` share - a split-K scratch per (device, stream), a status word per device - as the host keeps
them, with tensors in host memory and a recorder in the place of the native call path (nothing here reaches a GPU)."""
import contextlib
import threading
import types
import weakref

import pytest
import torch

from fp6_marlin_b200 import api

DEV, STREAM = torch.device("cuda", 63), 7
SMALL, LARGE = (1, 1024, 1024, 0), (128, 8192, 8192, 256)          # M, N, K, FP6 columns


@pytest.fixture
def registered(monkeypatch):
    """What `_device_buffers` registers with the native call path: ("scratch" or "device", arguments)."""
    calls, zeros = [], torch.zeros
    monkeypatch.setattr(api, "_call", types.SimpleNamespace(set_scratch=lambda *a: calls.append(("scratch", a)), set_device=lambda *a: calls.append(("device", a))))
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda index: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(torch, "zeros", lambda *args, device=None, **kw: zeros(*args, **kw))
    for name in ("_scratch", "_status", "_sm_count", "_scratch_need"):
        monkeypatch.setattr(api, name, {})
    return calls


def test_a_replaced_scratch_stays_alive(registered):
    """Another thread's call may have the address of the scratch and not have launched yet, and a captured graph keeps it."""
    _, first, _ = api._device_buffers(DEV, SMALL, STREAM)
    alive, size = weakref.ref(first), first.numel()
    assert registered[-1] == ("scratch", (63, STREAM, first.data_ptr(), size))
    del first
    _, second, _ = api._device_buffers(DEV, LARGE, STREAM)
    assert alive() is not None and alive() is not second
    assert registered[-1] == ("scratch", (63, STREAM, second.data_ptr(), second.numel()))
    assert api._device_buffers(DEV, SMALL, STREAM)[1] is second          # the larger one serves both from now on


def test_replaced_scratches_are_bounded(registered):
    """However a stream's calls grow, all its buffers are less than twice the last."""
    last = None
    for m in range(1, 1200, 7):
        for n in (1024, 4096, 8192):
            _, last, _ = api._device_buffers(DEV, (m, n, 4096, 0), STREAM)
    buffers = api._scratch[63, STREAM]
    assert buffers[-1] is last and sum(b.numel() for b in buffers) < 2 * last.numel()


def test_first_calls_of_two_threads_share_their_buffers(registered, monkeypatch):
    """Both threads reach the allocations of a stream's first call together (as far as they are let): one scratch and one status
    word are made, and what is registered is what both use."""
    together, zeros = threading.Barrier(2), torch.zeros
    made, got = [], []

    def slow_zeros(*args, **kw):
        with contextlib.suppress(threading.BrokenBarrierError):
            together.wait(0.3)
        made.append(zeros(*args, **kw))
        return made[-1]

    monkeypatch.setattr(torch, "zeros", slow_zeros)
    threads = [threading.Thread(target=lambda: got.append(api._device_buffers(DEV, SMALL, STREAM))) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 2 and len(registered) == 2
    (_, scratch, status), (_, other_scratch, other_status) = got
    assert scratch is other_scratch and status is other_status
    assert dict(registered) == {"device": (63, status.data_ptr(), 148), "scratch": (63, STREAM, scratch.data_ptr(), scratch.numel())}
