"""The one-pass quantise-and-pack kernels against the separate operations (torch quantisers, FP6 cast, packing
kernels) that ``make_w46_weight`` runs when the dequantised weight is wanted as well: same bytes for every form."""
import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import synth

pytestmark = pytest.mark.gpu


def _same(w, qc, gs):
    ref = fm.make_w46_weight(w, qc, gs, keep_dequantized=True, quant_device="cuda")
    got = fm.make_w46_weight(w, qc, gs, keep_dequantized=False, quant_device="cuda")
    assert torch.equal(got.B, ref.B)
    assert torch.equal(got.s.view(torch.int16), ref.s.view(torch.int16))


@pytest.mark.parametrize("k,n,qc,gs", [
    (128, 8, -1, 128), (128, 8, 8, 128), (256, 128, 128, 128), (256, 136, 8, 128), (384, 1312, 32, 128),
    (128, 131, 5, 128), (128, 130, 5, 128), (130, 257, 33, -1), (1, 1, -1, -1), (7, 300, 300, -1), (100, 64, 64, 128),
    (192, 320, 64, -1), (1024, 1280, 0, 128), (2048, 768, 200, -1),
])
def test_same_bytes_as_the_separate_operations(k, n, qc, gs):
    w = synth.make_weight_fp16(k, n, max(qc, 0), seed=k + n).to("cuda")
    _same(w, qc, gs)
    _same(w.t().contiguous().t(), qc, gs)                                # column-major input
    odd = torch.empty(k * n + 1, dtype=torch.float16, device="cuda")[1:].view(k, n)
    _same(odd.copy_(w), qc, gs)                                          # rows that start on no 4-byte boundary


@pytest.mark.parametrize("gs", [128, -1])
def test_every_half_as_the_maximum_and_special_values(gs):
    """Every non-negative half - subnormals, infinity and NaN among them - as a column's largest value, beside values
    of its own size, zero and smaller ones."""
    top = torch.arange(0, 1 << 15, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.float16)
    gen = torch.Generator(device="cuda").manual_seed(1)
    w = (torch.rand((128, top.numel()), generator=gen, device="cuda") * 2 - 1) * top.float()
    w = w.half()
    w[5] = top
    w[6] = 0
    w[7] = -top
    _same(w, -1, gs)


@pytest.mark.parametrize("value", [0.0, float("inf"), float("nan")])
def test_fp6_columns_that_cannot_be_coded_raise(value):
    w = synth.make_weight_fp16(256, 256, 64, seed=3).to("cuda")
    if value == 0.0:
        w[:, 200] = 0
    else:
        w[100, 200] = value
    for keep in (True, False):
        with pytest.raises(ValueError):
            fm.make_w46_weight(w, 64, 128, keep_dequantized=keep, quant_device="cuda")
    w[:, 200] = 2.0 ** -24                                               # a scale that rounds to zero: codes of +-28
    _same(w, 64, 128)
