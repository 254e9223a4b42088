"""The kernels for up to 8 and for 9 to 32 rows where their tiles, sets, teams and slices can go wrong: rows at both ends of every
instance, half a block at the end of K, strips narrower than 128 columns, slices shorter than the number of teams or sets, strips
cut over many CTAs and many strips in one CTA.

Bound: with operands that are exact (FP6: the dequantised weight of the oracle's rule; INT4 per group: the code times the scale in
fp32) all that remains beside fp32 sums is the rounding of the result to fp16, at most 2^-11 of a value, 2.1e-4 on average
over a binade; the dequantised INT4 weights it is compared with carry one more rounding of that size: 3e-4, and 1e-3 is asserted
for the worst row, as in the other tests."""
import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-3

# K, N, FP6 columns, group, CTAs offered
LAYERS = [
    (128, 256, 128, 128, -1),          # one block per strip
    (192, 512, 264, -1, -1),           # half a block at the end of K, ragged strips in both regions
    (384, 768, 40, 128, 1),            # every strip in one CTA, three blocks each: slices of fewer segments than teams
    (640, 512, 512, -1, 2),            # FP6 only; a boundary inside a strip
    (8192, 256, 72, 128, -1),          # strips cut over many CTAs
    (2048, 2304, 256, 128, 7),         # many strips per CTA, boundaries anywhere
]


@pytest.mark.parametrize("layer", LAYERS, ids=lambda v: "x".join(map(str, v)))
def test_rows_close_and_repeatable(layer):
    k, n, qc, group, sms = layer
    dev = torch.device("cuda", 0)
    w = synth.make_layer(k, n, qc, group, seed=k + n, keep_dequantized=False).to(dev)
    w64 = fm.dump_operands(w.B, w.s, k, n, qc, group).double()
    workspace = torch.zeros(n // 128 * 16, dtype=torch.int32, device=dev)
    for m in (1, 2, 7, 8, 9, 15, 16, 17, 31, 32):
        a = synth.make_activations(m, k, m).to(dev)
        residual = synth.make_activations(m, n, m + 1).to(dev)
        c = torch.full((m + 1, n), 3.0, dtype=torch.float16, device=dev)
        args = (w.s, workspace, qc)
        fm.mul(a, w.B, c[:m], *args, 64, 256, sms=sms, group_size=group, layout="b200")
        ref = a.double() @ w64
        assert (torch.linalg.norm(c[:m].double() - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max().item() <= TOL, m
        assert bool((c[m] == 3.0).all())
        again = torch.empty_like(c[:m])
        fm.mul(a, w.B, again, *args, 64, 256, sms=sms, group_size=group, layout="b200")
        assert torch.equal(again, c[:m]), "sums are added in one order"
        if k % 128:
            continue                        # (mul_fused takes the default tile shapes)
        fm.mul_fused(a, w.B, again, *args, epilogue="residual", residual=residual, sms=sms, group_size=group)
        ref = ref + residual.double()
        assert (torch.linalg.norm(again.double() - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max().item() <= TOL, m
    assert fm.device_status(dev) == 0
