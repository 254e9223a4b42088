"""9 to 32 rows on layers whose strips are cut over many CTAs: all teams and the warps before them sum a strip (gemm_team.cu).

Bound of the values: as in test_gpu_few_rows.py.  Bound of the time: against 8 rows, which another kernel serves, a call reads and sums two and four times the partials and streams the
same weights, which are most of it.  On 16384 x 1024 summing with two teams took 1.36 times the time at 16 rows and 2.0 times at 32
(9.1, 12.4 and 18.3 us), with four groups of warps 1.17 and 1.56 times; 1.27 and 1.75 are asserted."""
import pytest
import torch

import fp6_marlin_b200 as fm
from fp6_marlin_b200 import synth

pytestmark = pytest.mark.gpu
K, N = 8192, 256
TOL = 1e-3


@pytest.mark.parametrize("qc,group", [(72, 128), (136, -1)])
@pytest.mark.parametrize("sms", [2, 3, 5, 7, 11, 16])
def test_sums_of_shared_strips(qc, group, sms):
    """One to nine CTAs per strip, odd and even numbers of contributors, ragged strips, every epilogue."""
    dev = torch.device("cuda", 0)
    w = synth.make_layer(K, N, qc, group, seed=sms, keep_dequantized=False).to(dev)
    w64 = fm.dump_operands(w.B, w.s, K, N, qc, group).double()
    workspace = torch.zeros(N // 128 * 16, dtype=torch.int32, device=dev)
    for m in (9, 13, 16, 17, 24, 25, 32):
        a = synth.make_activations(m, K, m).to(dev)
        ref = a.double() @ w64
        c = torch.full((m + 1, N), 3.0, dtype=torch.float16, device=dev)
        fm.mul(a, w.B, c[:m], w.s, workspace, qc, sms=sms, group_size=group, layout="b200")
        assert (torch.linalg.norm(c[:m].double() - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max().item() <= TOL, m
        assert bool((c[m] == 3.0).all())
        again = synth.make_activations(m, N, m + 1).to(dev)
        ref = ref + again.double()
        fm.mul_fused(a, w.B, again, w.s, workspace, qc, epilogue="residual", residual=again, sms=sms, group_size=group)
        assert (torch.linalg.norm(again.double() - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max().item() <= TOL, m
        gate_up = torch.empty((m, N // 2), dtype=torch.float16, device=dev)
        fm.mul_fused(a, w.B, gate_up, w.s, workspace, qc, epilogue="silu_mul", sms=sms, group_size=group)
        sums = a.double() @ w64
        ref = torch.nn.functional.silu(sums[:, 0::2]) * sums[:, 1::2]
        assert (torch.linalg.norm(gate_up.double() - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max().item() <= 2 * TOL, m
    assert fm.device_status(dev) == 0


def _us_per_gemm(m, layers, s, workspace, k, n, qc):
    a, c = synth.make_activations(m, k, m).cuda(), torch.empty((m, n), dtype=torch.float16, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()

    def chain():
        for b in layers:
            fm.mul(a, b, c, s, workspace, qc, group_size=128, layout="b200")

    with torch.cuda.stream(stream):
        chain()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            chain()
        times = []
        for _ in range(14):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            graph.replay()
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end) * 1e3 / len(layers))
    return sorted(times[4:])[5]


@pytest.mark.parametrize("m,bound", [(16, 1.27), (32, 1.75)])
def test_time_on_a_narrow_layer(m, bound):
    """Sixteen CTAs per strip, weights larger than L2."""
    k, n, qc = 16384, 1024, 256
    w = synth.make_layer(k, n, qc, 128, seed=1, keep_dequantized=False).to(torch.device("cuda", 0))
    layers = [w.B.clone() for _ in range(32)]
    workspace = torch.zeros(n // 128 * 16, dtype=torch.int32, device="cuda")
    assert _us_per_gemm(m, layers, w.s, workspace, k, n, qc) <= bound * _us_per_gemm(8, layers, w.s, workspace, k, n, qc)
