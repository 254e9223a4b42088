"""Finished rows of the kernel for more than 128 rows leave through two buffers per team in shared memory, by tensor stores (full
strips) or 16-byte stores (ragged strips).  The sums have a fixed order, so the bits are those of the same launch with 2-byte
stores, which uses no buffer: an output whose rows are no multiples of 16 bytes."""
import ctypes

import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu


def _scatter(a, w, outputs, ld, n, qc, workspace, scratch, dev):
    table = (ctypes.c_void_p * len(outputs))(*[t.data_ptr() for t in outputs])
    m, k = a.shape
    rc = _lib.lib.fp6m_mul_scatter(a.data_ptr(), w.B.data_ptr(), table, len(outputs), ld, 0, n - max(qc, 0), w.s.data_ptr(), m, n, k,
                                   workspace.data_ptr(), workspace.numel() * 4, scratch.data_ptr(), scratch.numel(), dev.index,
                                   torch.cuda.current_stream(dev).cuda_stream, -1, -1, -1, 16, qc, 128, _lib.LAYOUT_B200, None)
    assert rc == _lib.OK


@pytest.mark.parametrize("m,k,n,qc", [
    (777, 256, 2048, 128),            # nine tiles of 96 rows: full strips, five blocks of the last tile beyond the last row
    (777, 256, 2048, 96),             # a ragged strip at the end of both regions, a full one before and behind it
    (300, 384, 2304, 32), (257, 128, 1024, 1000), (600, 512, 4096, -1), (1030, 256, 1280, 200),
])
@pytest.mark.parametrize("n_out", [0, 1, 8])
def test_same_bits_as_plain_stores(m, k, n, qc, n_out):
    dev = torch.device("cuda", 0)
    w = synth.make_layer(k, n, qc, 128, seed=m, keep_dequantized=False).to(dev)
    workspace = torch.zeros(n // 128 * 16, dtype=torch.int32, device=dev)
    _, scratch, _ = api._device_buffers(dev, (m, n, k, qc))
    assert fm.launch_plan(m, n, k, qc, torch.cuda.get_device_properties(dev).multi_processor_count) == (1, True)
    for seed in range(3):
        a = synth.make_activations(m, k, seed).to(dev)
        plain = torch.full((m, n + 1), 3.0, dtype=torch.float16, device=dev)
        _scatter(a, w, [plain], n + 1, n, qc, workspace, scratch, dev)
        runs = []
        for _ in range(12):                       # back to back, the outputs apart: nothing waits between the launches
            outs = [torch.full((m + 1, n), 3.0, dtype=torch.float16, device=dev) for _ in range(max(n_out, 1))]
            if n_out:
                _scatter(a, w, outs, n, n, qc, workspace, scratch, dev)
            else:
                fm.mul(a, w.B, outs[0][:m], w.s, workspace, qc, group_size=128, layout="b200")
            runs += outs
        torch.cuda.synchronize()
        for out in runs:
            assert torch.equal(out[:m], plain[:, :n])
            assert bool((out[m] == 3.0).all())
    assert fm.device_status(dev) == 0
