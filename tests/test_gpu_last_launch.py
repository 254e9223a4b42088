"""The last of several launches of the kernel for more than 128 rows goes to the kernel for up to 128 rows when it has no more
rows than that: its offsets of C, of the residual and of scattered outputs, next to a last launch that stays."""
import ctypes

import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu
K = 16384                                   # 2048 rows per launch: 64 MB of activations
TOL = 1e-3


@pytest.fixture(scope="module", params=[(512, 128), (768, 264)])
def layer(request):
    n, qc = request.param
    dev = torch.device("cuda", 0)
    w = synth.make_layer(K, n, qc, 128, seed=n, keep_dequantized=False).to(dev)
    workspace = torch.zeros(n // 128 * 16, dtype=torch.int32, device=dev)
    return w, workspace, fm.dump_operands(w.B, w.s, K, n, qc, 128).double()


def _rows_close(got, ref):
    assert (torch.linalg.norm(got.double() - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max().item() <= TOL


@pytest.mark.parametrize("m", [2049, 2100, 2176, 2177])
def test_epilogues_and_scattered_outputs(m, layer):
    w, workspace, w64 = layer
    n, qc, dev = w.n, w.quant_cols, w.B.device
    assert fm.launch_plan(m, n, K, qc, torch.cuda.get_device_properties(dev).multi_processor_count) == (2, True)
    a = synth.make_activations(m, K, m).to(dev)
    product = a.double() @ w64

    residual = torch.randn((m, n), generator=torch.Generator(device=dev).manual_seed(m), device=dev).half() * 4
    c = torch.full((m + 1, n), 3.0, dtype=torch.float16, device=dev)
    fm.mul_fused(a, w.B, c[:m], w.s, workspace, qc, epilogue="residual", residual=residual, group_size=128)
    _rows_close(c[:m], product + residual.double())
    assert bool((c[m] == 3.0).all())

    c = torch.full((m + 1, n // 2), 3.0, dtype=torch.float16, device=dev)
    fm.mul_fused(a, w.B, c[:m], w.s, workspace, qc, epilogue="silu_mul", group_size=128)
    gate, up = product[:, 0::2], product[:, 1::2]
    _rows_close(c[:m], gate * torch.sigmoid(gate) * up)
    assert bool((c[m] == 3.0).all())

    ld, col4, col6 = n + 512, 128, n + 512 - qc
    outs = [torch.full((m + 1, ld), 3.0, dtype=torch.float16, device=dev) for _ in range(2)]
    table = (ctypes.c_void_p * 2)(*[t.data_ptr() for t in outs])
    _, scratch, _ = api._device_buffers(dev, (m, n, K, qc))
    rc = _lib.lib.fp6m_mul_scatter(a.data_ptr(), w.B.data_ptr(), table, 2, ld, col4, col6, w.s.data_ptr(), m, n, K, workspace.data_ptr(),
                                   workspace.numel() * 4, scratch.data_ptr(), scratch.numel(), dev.index,
                                   torch.cuda.current_stream(dev).cuda_stream, -1, -1, -1, 16, qc, 128, _lib.LAYOUT_B200, None)
    assert rc == _lib.OK
    for out in outs:
        _rows_close(torch.cat([out[:m, col4: col4 + n - qc], out[:m, col6:]], dim=1), product)
        assert bool((out[m] == 3.0).all()) and bool((out[:, :col4] == 3.0).all()) and bool((out[:, col4 + n - qc: col6] == 3.0).all())
    assert fm.device_status(dev) == 0
