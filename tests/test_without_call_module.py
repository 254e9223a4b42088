"""The package without its extension module `_call` (a torch built without CUDA, another Python, nothing but libfp6m.so built): host
functions work, GEMMs take the general path."""
import os
import subprocess
import sys
import types

import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import api, synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
import sys, types, torch
{before}
import fp6_marlin, fp6_marlin_cpu
from fp6_marlin_b200 import api
assert isinstance(api._call, api._GeneralPathOnly), api._call
w = fp6_marlin.quantize(torch.linspace(0.0625, 28, 256 * 256).half().reshape(256, 256))
assert torch.equal(fp6_marlin_cpu.prepacking_cpu(w), fp6_marlin.prepacking(w))
print(w.view(torch.uint8).long().sum().item(), fp6_marlin.dequantize(w, torch.ones(256).half()).double().sum().item())
try:
    fp6_marlin.mul(*[torch.zeros(16, 128).half()] * 5)
except RuntimeError as e:
    assert "needs CUDA tensors" in str(e)
else:
    raise AssertionError
"""


@pytest.mark.parametrize("before", ["sys.modules['fp6_marlin_b200._call'] = None",
                                    "sys.modules['fp6_marlin_b200._call'] = types.SimpleNamespace(torch_version='0.1')"],
                         ids=["missing", "another torch"])
def test_host_functions(before):
    run = subprocess.run([sys.executable, "-c", PROGRAM.format(before=before)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr
    w = fm.quantize(torch.linspace(0.0625, 28, 256 * 256).half().reshape(256, 256))
    want = (w.view(torch.uint8).long().sum().item(), fm.dequantize(w, torch.ones(256).half()).double().sum().item())
    assert tuple(float(x) for x in run.stdout.split()) == want


@pytest.mark.gpu
def test_gemms(monkeypatch):
    k, n, qc = 512, 768, 264
    dev = torch.device("cuda", 0)
    w = synth.make_layer(k, n, qc, 128, seed=6, keep_dequantized=False).to(dev)
    a, residual = synth.make_activations(9, k, 1).to(dev), synth.make_activations(9, n, 2).to(dev)
    workspace = torch.zeros(n // 128 * 16, dtype=torch.int32, device=dev)

    def both():
        c, r = torch.zeros((9, n), dtype=torch.float16, device=dev), torch.zeros((9, n), dtype=torch.float16, device=dev)
        fm.mul(a, w.B, c, w.s, workspace, qc, group_size=128, layout="b200")
        fm.mul_fused(a, w.B, r, w.s, workspace, qc, epilogue="residual", residual=residual, group_size=128)
        return c, r

    want = both()
    assert isinstance(api._call, types.ModuleType)          # where there is a GPU, the module is built and used
    monkeypatch.setattr(api, "_call", api._GeneralPathOnly("of this test"))
    for name in ("_scratch", "_status", "_sm_count"):
        monkeypatch.setattr(api, name, {})
    with pytest.warns(RuntimeWarning, match="general path, because of this test"):
        got = both()
    torch.cuda.synchronize()
    assert all(torch.equal(p, q) for p, q in zip(want, got))
    assert fm.device_status(dev) == 0
