"""First calls of threads and of a process: every one of them works."""
import subprocess
import sys
import threading

import pytest
import torch

import fp6_marlin_b200 as fm
from conftest import ROOT
from fp6_marlin_b200 import synth

K, N = 256, 512
ROWS = [1, 20, 40, 100, 300, 16, 64, 129] * 2          # every kernel instance


def run_from_threads(warm_up):
    dev = torch.device("cuda", 0)
    w = synth.make_layer(K, N, 128, 128, seed=1, keep_dequantized=False).to(dev)
    jobs = []
    for m in ROWS:
        stream = torch.cuda.Stream(dev)
        with torch.cuda.stream(stream):
            c = torch.zeros((m, N), dtype=torch.float16, device=dev)
            fm.api._device_buffers(dev, (m, N, K, 128))
        jobs.append((synth.make_activations(m, K, m).to(dev), c, torch.zeros(N // 128 * 16, dtype=torch.int32, device=dev), stream))
    if warm_up:
        for a, c, workspace, _ in jobs:
            fm.mul(a, w.B, torch.empty_like(c), w.s, workspace, 128, group_size=128, layout="b200")
    torch.cuda.synchronize()
    go, failures = threading.Barrier(len(jobs)), []

    def work(a, c, workspace, stream):
        try:
            with torch.cuda.stream(stream):
                go.wait()
                fm.mul(a, w.B, c, w.s, workspace, 128, group_size=128, layout="b200")
        except Exception as e:
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failures, failures
    w64 = fm.dump_operands(w.B, w.s, K, N, 128, 128).double()
    for a, c, _, _ in jobs:
        ref = a.double() @ w64
        assert (torch.linalg.norm(c.double() - ref) / torch.linalg.norm(ref)).item() <= 1e-3


@pytest.mark.gpu
def test_first_call_of_a_thread():
    """A thread that has made no CUDA call has no current context, which the driver's tensor-map encoder needs."""
    run_from_threads(warm_up=True)


@pytest.mark.gpu
@pytest.mark.parametrize("attempt", range(3))
def test_first_calls_of_a_process_from_several_threads(attempt):
    """The tensor-map encoder, kernel attributes and multiprocessor counts are looked up on first use."""
    program = "import sys; sys.path[:0] = ['.', 'tests']; import test_gpu_first_calls as t; t.run_from_threads(warm_up=False); print('ok')"
    run = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip().endswith("ok"), run.stdout[-2000:] + run.stderr[-2000:]
