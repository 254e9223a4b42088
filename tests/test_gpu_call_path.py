"""The native call path of mul and mul_fused against the general one: plain CUDA tensors take the former, anything else the
latter, with the same results and the same errors."""
import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import api, synth

pytestmark = pytest.mark.gpu
K, N, QC = 512, 768, 264


class Subclass(torch.Tensor):
    pass


@pytest.fixture(scope="module")
def layer():
    return synth.make_layer(K, N, QC, 128, seed=5, keep_dequantized=False).to(torch.device("cuda", 0))


def _count_native(monkeypatch):
    calls = []
    native = api._call

    class Counting:
        def __getattr__(self, name):
            return getattr(native, name)

        def mul(self, *args):
            calls.append(native.mul(*args))
            return calls[-1]

    monkeypatch.setattr(api, "_call", Counting())
    return calls


@pytest.mark.parametrize("m", [1, 9, 32])           # sums in one order: the same bits
def test_same_results_on_both_paths(m, layer, monkeypatch):
    dev = layer.B.device
    a, residual = synth.make_activations(m, K, m).to(dev), synth.make_activations(m, N, m + 1).to(dev)
    workspace = torch.zeros(N // 128 * 16, dtype=torch.int32, device=dev)
    calls = _count_native(monkeypatch)
    out = []
    stream = torch.cuda.Stream(dev)                  # a stream of its own: the first call may create its scratch
    stream.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(stream):
        for x in (a, a, torch.nn.Parameter(a, requires_grad=False), a.as_subclass(Subclass)):
            c, r, s = (torch.full((m, n), 3.0, dtype=torch.float16, device=dev) for n in (N, N, N // 2))
            fm.mul(x, layer.B, c, layer.s, workspace, QC, group_size=128, layout="b200")
            fm.mul_fused(x, layer.B, r, layer.s, workspace, QC, epilogue="residual", residual=residual, group_size=128)
            fm.mul_fused(x, layer.B, s, layer.s, workspace, QC, epilogue="silu_mul", group_size=128)
            out.append((c, r, s))
    stream.synchronize()
    assert calls[0] in (-1, 0) and calls[1:] == [0] * 8 + [-1] * 3
    for other in out[1:]:
        assert all(torch.equal(p, q) for p, q in zip(out[0], other))


def test_same_errors(layer):
    dev = layer.B.device
    a, c = synth.make_activations(4, K, 1).to(dev), torch.zeros((4, N), dtype=torch.float16, device=dev)
    workspace = torch.zeros(N // 128 * 16, dtype=torch.int32, device=dev)

    def mul(a=a, c=c, workspace=workspace, **kw):
        fm.mul(a, layer.B, c, layer.s, workspace, QC, group_size=128, layout="b200", **kw)

    mul()
    for match, call in (("workspace must be of size at least", lambda: mul(workspace=workspace[:-1])),
                        ("must be float16", lambda: mul(a=a.float())), ("must be contiguous", lambda: mul(a=a.t().contiguous().t())),
                        ("as many rows as A", lambda: mul(c=c[:3])), ("not compatible with thread_k=96", lambda: mul(thread_k=96, thread_n=128)),
                        ("No kernel implementation", lambda: mul(thread_k=256, thread_n=256)), ("needs CUDA tensors", lambda: mul(a=a.cpu()))):
        with pytest.raises(RuntimeError, match=match):
            call()
    mul(a=a[:0], c=c[:0])                            # nothing to do
    assert fm.device_status(dev) == 0
